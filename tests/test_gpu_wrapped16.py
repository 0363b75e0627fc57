"""16-bit storage where an odd step's chunks wrap around the box or reflect from halfway walls (out of line
there, on a copy of the populations), and where nodes of x planes leave with their row, against the
FP64 oracle.  Bars: 2e-3 (FP16) and 2e-2 (BF16) of the largest velocity, those of
test_reduced_precision_vs_fp64_oracle.
"""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from nonnewlbm_b200 import CaseSpec, Lattice, capi
from nonnewlbm_b200 import geometry as G

pytestmark = pytest.mark.gpu
BAR = {"f16": 2e-3, "bf16": 2e-2}


def _velocities_agree(orc, lat, m, dtype):
    on = (m == G.MAP_FLUID) | (m == G.MAP_PERIODIC)
    pairs = [(orc.get_macro(fo)[on], lat.macro(fl)[on])
             for fo, fl in ((O.M_VX, capi.M_VX), (O.M_VY, capi.M_VY), (O.M_VZ, capi.M_VZ))]
    umax = max(np.max(np.abs(a)) for a, _ in pairs)
    for a, b in pairs:
        assert np.max(np.abs(a - b)) <= BAR[dtype] * umax


@pytest.mark.parametrize("collision", ["CUM", "KBC_N4"])
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("bounce_back", ["fullway", "halfway"])
@pytest.mark.parametrize("nx", [9, 33, 65])
def test_wrapped_rows(nx, bounce_back, dtype, collision):
    m = np.full((5, 6, nx), G.MAP_PERIODIC, dtype=np.uint8)
    m[1, 3, 6:8] = m[2, 2, nx - 2] = G.MAP_WALL
    if bounce_back == "halfway":
        m[0, 1:3, 2:4] = m[-1, 0, 5] = m[1:3, -1, 0] = m[3, 2, -1] = G.MAP_WALL
    orc = O.Oracle(nx, 6, 5, collision=O.COLLISIONS.index(collision), nu=0.03, halfway=bounce_back == "halfway")
    lat = Lattice(CaseSpec((nx, 6, 5), collision=collision, dtype=dtype, nu=0.03, bounce_back=bounce_back))
    for L in (orc, lat):
        L.set_map(m)
        L.init_equilibrium(1.001, 0.02, -0.01, 0.015)
    orc.step(17)
    lat.step(17, macro=True)
    _velocities_agree(orc, lat, m, dtype)


@pytest.mark.parametrize("cells", [1, 2])
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("nx", [31, 32, 33, 65])
def test_box_rows(nx, dtype, cells):
    m, prof = G.dense_box_map(nx, 7, 6)
    orc = O.Oracle(nx, 7, 6, collision=0, nu=0.02)
    lat = Lattice(CaseSpec((nx, 7, 6), collision="CUM", dtype=dtype, nu=0.02))
    orc.set_map(m)
    orc.set_inflow_profile(G.expand_profile(m, prof) * 0.04)
    lat.set_map(m)
    lat.set_inflow_profile(prof * 0.04)
    lat.set_launch(64, cells)
    for L in (orc, lat):
        L.init_equilibrium(1.001, 0.01, -0.005, 0.004)
    orc.step(41)                       # a graph of 16 steps twice and nine steps more
    lat.step(41, macro=True)
    _velocities_agree(orc, lat, m, dtype)
