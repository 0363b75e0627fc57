"""A GEO_INFLOW node whose neighbour at x + 1 is the only serving cell of its chunk and has another open-plane
node beside it, against the FP64 C oracle (1e-12 relative per population, the bar of the other
parity tests).  Both nodes are written by that one cell's warp.
"""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from nonnewlbm_b200 import CaseSpec, Lattice, capi
from nonnewlbm_b200 import geometry as G

from helpers import dead_mask, max_rel

pytestmark = pytest.mark.gpu


def _map(kind):
    if kind == "one_cell_rows":        # inlet, one fluid cell, outlet: rows of three cells
        return G.pipe_map(3, 16, 16, 6.0)[0]
    m = np.full((6, 8, 12), G.MAP_WALL, dtype=np.uint8)
    m[1:5, 1:7, 4:11] = G.MAP_FLUID    # starts on a 32-byte boundary: the inlet at x = 3 is outside the chunks
    m[1:5, 1:7, 3] = G.MAP_INFLOW_EQ
    if kind == "front":
        m[1:5, 0, 4] = G.MAP_OUTFLOW_FRONT
    else:
        m[1:5, 7, 4] = G.MAP_OUTFLOW_BACK
    return m


@pytest.mark.parametrize("bounce_back", ["fullway", "halfway"])
@pytest.mark.parametrize("kind", ["one_cell_rows", "front", "back"])
def test_fp64_inlet_beside_another_node(kind, bounce_back):
    m = _map(kind)
    nz, ny, nx = m.shape
    n_in = int((m == G.MAP_INFLOW_EQ).sum())
    prof = np.column_stack([0.02 + 0.001 * np.arange(n_in) / n_in, np.full(n_in, 0.002), np.full(n_in, -0.001)])
    orc = O.Oracle(nx, ny, nz, collision=0, nu=0.03, halfway=bounce_back == "halfway")
    lat = Lattice(CaseSpec((nx, ny, nz), collision="CUM", dtype="f64", nu=0.03, bounce_back=bounce_back))
    orc.set_map(m)
    orc.set_inflow_profile(G.expand_profile(m, prof))
    lat.set_map(m)
    lat.set_inflow_profile(prof)
    for L in (orc, lat):
        L.init_equilibrium(1.001, 0.01, -0.005, 0.004)
    live = np.broadcast_to(m != G.MAP_WALL, (27,) + m.shape) if bounce_back == "halfway" else ~dead_mask(m)
    for n in (1, 2, 4):                # ends in either A-A layout
        orc.step(n)
        lat.step(n, macro=True, reduce=True)
        assert max_rel(lat.export_df()[live], orc.get_df()[live]) <= 1e-12, n
    on = m != G.MAP_WALL
    for fo, fl in ((O.M_RHO, capi.M_RHO), (O.M_VX, capi.M_VX), (O.M_VY, capi.M_VY)):
        assert np.max(np.abs(lat.macro(fl) - orc.get_macro(fo))[on]) <= 1e-13
    assert np.max(np.abs(lat.reduce() - orc.reduce())) <= 1e-10 * abs(orc.reduce()[0])
