"""The stored values of 16-bit runs, bit for bit.

A value next to a rounding boundary of the 16-bit type is stored one unit away by any other order
of the same FP32 operations, and the steps after it carry that on, so a run that is continued or
compared with a stored one needs the same order.  The digests are of the populations and the
velocity after 41 steps (a graph of 16 steps twice and nine steps more) on one B200; they were
taken before the collisions of FP32 and FP64 storage were put on the stored values.
"""
from __future__ import annotations

import hashlib

import numpy as np
import pytest

from nonnewlbm_b200 import CaseSpec, Lattice, capi
from nonnewlbm_b200 import geometry as G

from helpers import dead_mask, small_junction

pytestmark = pytest.mark.gpu
CY = (0.05, 40.0, 2.0, 0.3568)

# collision/storage/cells a thread/options: digest
DIGESTS = {
    "CUM/f16/1": "9ff5dda22b863326",
    "CUM/f16/2": "8e651ce4e7eb6797",
    "BGK/f16/1": "bf7ca830c033b0c9",
    "BGK/f16/2": "83e795b18a8975ce",
    "MRT_LES/f16/1": "37e6f9bca4e50487",
    "MRT_LES/f16/2": "abbd6c839d4a8e45",
    "KBC_N1/f16/1": "dda219f5800d6f1c",
    "KBC_N4/f16/1": "3d3b2d67b4450e52",
    "KBC_C4/f16/1": "b4a5c0e414594611",
    "CUM/bf16/1": "3d311d93322e1939",
    "CUM/bf16/2": "75c5a9fc66fb17cb",
    "BGK/bf16/1": "eb06fc145bbe37c1",
    "BGK/bf16/2": "9489386e6fd92251",
    "MRT_LES/bf16/1": "a574d261f8d361a8",
    "MRT_LES/bf16/2": "0bfe11e27c1f1a84",
    "KBC_N1/bf16/1": "4208777562b6c194",
    "KBC_N4/bf16/1": "09a75e19c19eb30b",
    "KBC_C4/bf16/1": "dc2a2fccd51325ab",
    "CUM/f16/1/cy": "de2d6bcb1b6de0aa",
    "CUM/f16/2/cy": "045ab1f77b78e9c0",
    "KBC_N4/f16/1/cy": "c1491ab5d3f925be",
    "MRT_LES/bf16/1/cy": "7f568d340f340c52",
    "BGK/bf16/2/cy": "5ecf73314a578c67",
    "KBC_C2/f16/1/cy": "5309d950b02104fb",
    "KBC_N3/bf16/1": "cfff0764597c65b9",
    "CUM/f16/1/box": "383805229b8fd937",
    "CUM/bf16/2/box": "9b7ea8e73cd3e794",
    "BGK/bf16/1/box": "74c59c3f56a494bb",
    "MRT_LES/f16/1/box": "bfa829c33b12ab4d",
    "KBC_N4/f16/1/box": "cb5514ea4abdeaf4",
    "MRT_LES/f16/1/halfway": "14414c403598ae40",
    "CUM/f16/2/halfway": "c1a7e5f4d335da33",
    "KBC_N4/bf16/1/halfway": "c06089b868d70610",
    "BGK/f16/1/force": "1857c001a4e18717",
    "KBC_N4/f16/1/force": "95faa65efdae3bc0",
    "CUM/bf16/1/force": "714e51e83be7f935",
    "MRT_LES/f16/2/force": "933d12645e92c139",
}


def _digest(name: str) -> str:
    collision, dtype, cells, *opts = name.split("/")
    kw = {"cy_mode": "local-neq", "cy": CY} if "cy" in opts else {}
    if "halfway" in opts:
        kw["bounce_back"] = "halfway"
    if "force" in opts:
        kw["force"] = (2e-5, -1e-5, 1.5e-5)
    if "box" in opts:                  # nodes of x planes in the rows, rows on the faces
        m, prof = G.dense_box_map(40, 7, 6)
        lat = Lattice(CaseSpec((40, 7, 6), collision=collision, dtype=dtype, nu=0.02, **kw))
        lat.set_map(m)
        lat.set_inflow_profile(prof * 0.04)
    else:
        wall = small_junction()
        lat = Lattice(CaseSpec(wall.shape[::-1], collision=collision, dtype=dtype, nu=0.02, **kw))
        a = lat.setup_tcpc(wall)
        lat.set_inflow(ivc_flux=0.03 * a["left_area"], svc_flux=0.02 * a["right_area"])
        m = capi.tcpc_labels(wall)[0]
    lat.set_launch(64, int(cells))
    lat.init_equilibrium(1.001, 0.01, -0.005, 0.004)
    lat.step(41, macro=True)
    live = np.broadcast_to(m != G.MAP_WALL, (27,) + m.shape) if "halfway" in opts else ~dead_mask(m)
    h = hashlib.sha256(np.ascontiguousarray(lat.export_df()[live], dtype=np.float32).tobytes())
    for f in (capi.M_RHO, capi.M_VX, capi.M_VY, capi.M_VZ):
        h.update(np.ascontiguousarray(lat.macro(f)[m == G.MAP_FLUID], dtype=np.float32).tobytes())
    lat.close()
    return h.hexdigest()[:16]


@pytest.mark.parametrize("name", DIGESTS)
def test_stored_values(name):
    assert _digest(name) == DIGESTS[name]
