"""Odd-step addresses of chunks next to a face or a halfway wall.  Bar: 1e-12
relative per population against the FP64 oracle, the bar of the other parity tests.
"""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from nonnewlbm_b200 import CaseSpec, Lattice
from nonnewlbm_b200 import geometry as G

from helpers import dead_mask, max_rel

pytestmark = pytest.mark.gpu


def _torus(nx, ny, nz, face_walls):
    """All periodic, with walls inside and (`face_walls`) on faces and an edge."""
    m = np.full((nz, ny, nx), G.MAP_PERIODIC, dtype=np.uint8)
    m[1, 3, 6:8] = m[2, 2, nx - 2] = G.MAP_WALL
    if face_walls:
        m[0, 1:3, 2:4] = m[-1, 0, 5] = m[1:3, -1, 0] = m[3, 2, -1] = G.MAP_WALL
    return m


@pytest.mark.parametrize("bounce_back", ["fullway", "halfway"])
@pytest.mark.parametrize("nx", [9, 32, 33, 65])
def test_fp64_wrapped_rows(nx, bounce_back):
    m = _torus(nx, 6, 5, bounce_back == "halfway")
    orc = O.Oracle(nx, 6, 5, collision=0, nu=0.03, halfway=bounce_back == "halfway")
    lat = Lattice(CaseSpec((nx, 6, 5), collision="CUM", dtype="f64", nu=0.03, bounce_back=bounce_back))
    for L in (orc, lat):
        L.set_map(m)
        L.init_equilibrium(1.001, 0.02, -0.01, 0.015)
    live = np.broadcast_to(m != G.MAP_WALL, (27,) + m.shape) if bounce_back == "halfway" else ~dead_mask(m)
    for n in (1, 2, 4, 17):            # ends in either A-A layout
        orc.step(n)
        lat.step(n)
        assert max_rel(lat.export_df()[live], orc.get_df()[live]) <= 1e-12, n
