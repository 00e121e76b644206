"""Cycles that are kept on grids whose coarse levels are dense matrices (mgp_kernels.cu,
TinyLv): as test_gpu_tiny_levels, with right-hand sides whose residual every cycle lowers, so
that what is compared with the oracle is three V-cycles and not a correction taken back."""
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


@pytest.mark.parametrize("kind", ["mg", "dd"])
@pytest.mark.parametrize("nx,ny", [(8, 8), (12, 6), (16, 16), (24, 8), (32, 16)])
@pytest.mark.parametrize("types", [[D, D, D, D], [D, D, N, N], [P, P, D, D], [D, D, P, P]])
def test_three_cycles_follow_the_oracle(M, kind, nx, ny, types):
    v = Box.of_size(nx, ny)
    geo = G.mapped_geometry(v, G.map_identity())
    rhs = BoxData(v)
    rhs.data[:] = np.random.default_rng(nx * 100 + ny).standard_normal(rhs.data.shape)
    bc = BdryData(v, types, [BCMODE_UNIFORM] * 4)
    dd = kind == "dd"
    O.lib().or_set_dirichlet_coupled_diagonal.argtypes = [ctypes.c_int]
    O.lib().or_set_dirichlet_coupled_diagonal(1)
    po, pd = BoxData(v, 1, 1), BoxData(v, 1, 1)
    try:
        ro = (O.dc_vcycle if dd else O.vcycle)(po, rhs.copy(), geo, bc, True, 1e-30, 3, smooth_down=4, smooth_up=4,
                                               smooth_bottom=4, gs_order=1)
    finally:
        O.lib().or_set_dirichlet_coupled_diagonal(0)
    with M.Solver(v, geo, bc, KIND_DD if dd else KIND_MG, M.FLAG_DIRICHLET_COUPLED_DIAG) as s:
        rd = (s.dc_vcycle if dd else s.vcycle)(pd, rhs.copy(), bc, True, 1e-30, 3, 1, 4, 4, 4)
    assert ro.iterations == rd.iterations == 3 and not ro.diverged and not rd.diverged
    a, b = po.interior(), pd.interior()
    # as test_gpu_tiny_levels: rounding of sums in another order through BiCGStab to 1e-6 on some tens of cells
    assert np.abs(a).max() > 0 and np.abs(a - b).max() <= 1e-10 * np.abs(a).max()
