"""Open-plane nodes of x planes, which leave with their row's own stores where they are lanes of a
plain chunk, against the FP64 C oracle.

The row widths put the outlet node in the last lane of a chunk, in the first lane of none
(one cell past a chunk) and inside one; rows on the y and z faces, a second inlet node in
the same chunk and rows behind walls take the other paths.  Bars: FP64 1e-12 relative per
population, the bar of the other parity tests; FP32 2e-5 of the largest velocity, the
bar of test_fp32_collisions_vs_fp64_oracle.
"""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from nonnewlbm_b200 import CaseSpec, Lattice, capi
from nonnewlbm_b200 import geometry as G

from helpers import dead_mask, max_rel

pytestmark = pytest.mark.gpu


def _box(nx, ny, nz, variant):
    m, prof = G.dense_box_map(nx, ny, nz)
    if variant == "two_inlets":        # a second inlet plane inside the rows: two nodes in one chunk
        m[:, :, 9] = G.MAP_INFLOW_EQ
        prof = np.zeros((2 * ny * nz, 3))
        prof[:, 0] = 1.0
        prof[1::2, 1] = 0.3            # the two nodes of a row differ
    elif variant == "walls":           # a duct: no row on a face, no gathered node
        m[m == G.MAP_PERIODIC] = G.MAP_FLUID
        m[0] = m[-1] = G.MAP_WALL
        m[:, 0] = m[:, -1] = G.MAP_WALL
        m[2, 3, 0] = G.MAP_WALL        # and a hole in the inlet plane
        prof = prof[:int((m == G.MAP_INFLOW_EQ).sum())]
    return m, prof


def _pair(m, prof, collision, dtype, eq="inv_cum_ref"):
    nz, ny, nx = m.shape
    orc = O.Oracle(nx, ny, nz, collision=O.COLLISIONS.index(collision), equilibrium=capi.EQUILIBRIA[eq], nu=0.02)
    lat = Lattice(CaseSpec((nx, ny, nz), collision=collision, dtype=dtype, equilibrium=eq, nu=0.02))
    orc.set_map(m)
    orc.set_inflow_profile(G.expand_profile(m, prof) * 0.04)
    lat.set_map(m)
    lat.set_inflow_profile(prof * 0.04)
    for L in (orc, lat):
        L.init_equilibrium(1.001, 0.01, -0.005, 0.004)
    return orc, lat


@pytest.mark.parametrize("variant", ["plain", "two_inlets", "walls"])
@pytest.mark.parametrize("nx", [31, 32, 33, 34, 64, 65])
def test_fp64_box_rows(nx, variant):
    m, prof = _box(nx, 7, 6, variant)
    orc, lat = _pair(m, prof, "CUM", "f64")
    for n in (1, 2, 4):                # ends in either A-A layout
        orc.step(n)
        lat.step(n, macro=True, reduce=True)
        assert max_rel(lat.export_df(), orc.get_df(), dead_mask(m)) <= 1e-12, n
    for fo, fl in ((O.M_RHO, capi.M_RHO), (O.M_VX, capi.M_VX), (O.M_VY, capi.M_VY)):
        assert np.max(np.abs(lat.macro(fl) - orc.get_macro(fo))) <= 1e-13


@pytest.mark.parametrize("eq", ["inv_cum", "default", "entropic"])
def test_fp64_box_rows_equilibria(eq):
    m, prof = _box(34, 6, 5, "plain")
    orc, lat = _pair(m, prof, "BGK", "f64", eq)
    orc.step(9)
    lat.step(9)
    assert max_rel(lat.export_df(), orc.get_df(), dead_mask(m)) <= 1e-12


@pytest.mark.parametrize("nx", [32, 33, 48, 65])
def test_fp64_junction_rows(nx):
    """The IVC and SVC planes (IN_L, IN_R) of a junction."""
    wall = G.study_to_geometry(G.junction(nx, 26, 24, r_ivc=5, r_svc=4.5, r_chamber=6, r_out=4, z_offset=2))
    orc = O.Oracle(nx, 26, 24, collision=0, nu=0.02)
    lat = Lattice(CaseSpec((nx, 26, 24), collision="CUM", dtype="f64", nu=0.02))
    _, counts = orc.setup_tcpc(wall)
    lat.setup_tcpc(wall)
    for L in (orc, lat):
        L.set_inflow(ivc_flux=0.03 * counts[0], svc_flux=0.02 * counts[1])
        L.init_equilibrium()
    orc.step(25)
    lat.step(25, reduce=True)
    assert max_rel(lat.export_df(), orc.get_df(), dead_mask(orc.get_map())) <= 1e-12
    assert np.max(np.abs(lat.reduce() - orc.reduce())) <= 1e-10 * abs(orc.reduce()[0])


@pytest.mark.parametrize("cells", [1, 2])
@pytest.mark.parametrize("collision", ["CUM", "BGK", "MRT_LES"])
def test_fp32_box_rows(collision, cells):
    m, prof = _box(40, 7, 6, "plain")
    orc, lat = _pair(m, prof, collision, "f32")
    lat.set_launch(64, cells)
    orc.step(41)                       # graph of 16 steps twice and nine steps more
    lat.step(41, macro=True)
    umax = np.max(np.abs(orc.get_macro(O.M_VX)))
    for fo, fl in ((O.M_VX, capi.M_VX), (O.M_VY, capi.M_VY), (O.M_VZ, capi.M_VZ)):
        assert np.max(np.abs(lat.macro(fl) - orc.get_macro(fo))) <= 2e-5 * umax
