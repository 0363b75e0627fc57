"""Odd-step addresses of chunks next to a face or a halfway wall, and the phases of the
finite-difference Carreau-Yasuda coupling in each way that a kernel finds its case's arguments
(one case, up to 16 in the parameters, more in a device array).  Bars: 1e-12 relative per
population against the FP64 oracle, the bar of the other parity tests; a case of a batch is
bitwise the same case alone.
"""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from nonnewlbm_b200 import CaseSpec, Lattice
from nonnewlbm_b200 import geometry as G

from helpers import dead_mask, max_rel, small_junction

pytestmark = pytest.mark.gpu
CY = (0.05, 40.0, 2.0, 0.3568)


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


@pytest.mark.parametrize("bounce_back", ["fullway", "halfway"])
@pytest.mark.parametrize("n_cases", [1, 2, 17])
def test_ref_fd_batch_is_the_case_alone(n_cases, bounce_back):
    wall = small_junction()
    shape = wall.shape[::-1]

    def run(nus):
        lat = Lattice([CaseSpec(shape, collision="CUM", dtype="f64", cy_mode="ref-fd", nu=nu, cy=CY, bounce_back=bounce_back)
                       for nu in nus])
        for k in range(len(nus)):
            a = lat.setup_tcpc(wall, ic=k)
            lat.set_inflow(ivc_flux=0.03 * a["left_area"], svc_flux=0.02 * a["right_area"], ic=k)
            lat.init_equilibrium(ic=k)
        lat.step(35)                   # a chained graph twice and three steps more
        out = [lat.export_df(k) for k in range(len(nus))]
        lat.close()
        return out

    nus = [0.02 + 0.001 * k for k in range(n_cases)]
    batch = run(nus)
    for k in {0, n_cases - 1}:
        orc = O.Oracle(*shape, collision=0, nu=nus[k], cy_mode=O.CY_REF_FD, cy=CY, halfway=bounce_back == "halfway")
        rc, counts = orc.setup_tcpc(wall)
        orc.set_inflow(ivc_flux=0.03 * counts[0], svc_flux=0.02 * counts[1])
        orc.init_equilibrium()
        orc.step(35)
        m = orc.get_map()
        live = np.broadcast_to(m != G.MAP_WALL, (27,) + m.shape) if bounce_back == "halfway" else ~dead_mask(m)
        assert max_rel(batch[k][live], orc.get_df()[live]) <= 1e-12, k
        assert np.array_equal(batch[k][live], run([nus[k]])[0][live]), k
