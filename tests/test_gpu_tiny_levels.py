"""Coarse levels of at most 64 cells run as dense matrices in the staged coarse
cycle (mgp_kernels.cu, TinyLv): sweeps, the bottom's operator and BiCGStab's
preconditioner.  Grids small enough that these levels are most of the hierarchy,
at the edges of the range (4 x 4, 64 cells, one above), with every kind of side a
matrix covers -- among them Dirichlet beside Neumann sides, whose corner
closures read stored ghosts from the cycle before -- and two coarse visits.  (Not
four Neumann sides: the bottom operator is singular there, and BiCGStab's last
iterations on it amplify rounding in any order of summation.)"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from helpers import D, N, P
from mgpoisson2d_b200 import geometry as G
from mgpoisson2d_b200.types import BCMODE_UNIFORM, KIND_DD, KIND_MG, BdryData, Box, BoxData
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def M():
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as api
    return api


def _problem(nx, ny, types):
    v = Box.of_size(nx, ny)
    geo = G.mapped_geometry(v, G.map_skew_stretch(15.0, 1.02, 0.25, ny) if P not in types else G.map_identity())
    rng = np.random.default_rng(nx * 100 + ny)
    rhs = BoxData(v)
    rhs.data[:] = rng.standard_normal(rhs.data.shape)
    rhs.data -= rhs.data.mean()
    return v, geo, rhs, BdryData(v, types, [BCMODE_UNIFORM] * 4)


# The matrices sum in another order than the sweeps: a relative 64 * 2^-53 = 1e-14 an application, and BiCGStab to
# 1e-6 on a level of condition at most some hundreds carries a rounding into the correction by that factor and its few
# iterations: 1e-10 of the largest value leaves another factor of ten.
TOL = 1e-10


@pytest.mark.parametrize("kind", ["mg", "dd"])
@pytest.mark.parametrize("nx,ny", [(4, 4), (8, 8), (16, 4), (13, 5), (12, 6), (16, 16), (24, 8), (32, 16)])
@pytest.mark.parametrize("types", [[D, D, D, D], [D, D, N, N], [N, D, D, N], [N, N, N, D], [P, P, D, D], [D, N, P, P]])
def test_tiny_levels_follow_the_oracle(M, kind, nx, ny, types):
    v, geo, rhs, bc = _problem(nx, ny, types)
    dd = kind == "dd"
    O.lib().or_set_dirichlet_coupled_diagonal.argtypes = [ctypes.c_int]
    O.lib().or_set_dirichlet_coupled_diagonal(1)
    po, pd = BoxData(v, 1, 1), BoxData(v, 1, 1)
    try:
        ro = (O.dc_vcycle if dd else O.vcycle)(po, rhs.copy(), geo, bc, True, 1e-30, 3, numcycles=2, smooth_down=2,
                                               smooth_up=3, smooth_bottom=4, gs_order=1)
    finally:
        O.lib().or_set_dirichlet_coupled_diagonal(0)
    with M.Solver(v, geo, bc, KIND_DD if dd else KIND_MG, M.FLAG_DIRICHLET_COUPLED_DIAG) as s:
        rd = (s.dc_vcycle if dd else s.vcycle)(pd, rhs.copy(), bc, True, 1e-30, 3, 2, 2, 3, 4)
    if ro.iterations != rd.iterations or ro.diverged != rd.diverged:
        # only where both stand at rounding level may the residual grow in one and not in the other
        assert max(ro.relres[-1], rd.relres[-1]) < 1e-12
    a, b = po.interior(), pd.interior()
    assert np.abs(a - b).max() <= TOL * max(np.abs(a).max(), 1e-300)
