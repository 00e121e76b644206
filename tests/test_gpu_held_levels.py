"""The one-CTA coarse cycle sweeps its levels of more than 64 cells with the
windows of the sweep kernels (mgp_sweep.cuh, mgp_ddsweep.cuh).  Grids that are such
levels themselves, at the edges of each window and one past them, for the sides a
window covers: one V-cycle without a coarse visit (numcycles = 0) is the sweeps,
the residual and the prolonged guess, and has the oracle's bits."""
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


# windows: 32 x 48 and 64 x 24 (9-point), 32 x 64 and 64 x 32 (deferred correction)
SIZES = [(32, 32), (16, 48), (64, 16), (40, 24), (10, 50), (66, 14), (34, 26), (14, 64), (12, 66), (34, 30), (18, 4), (4, 18)]


@pytest.mark.parametrize("kind", ["mg", "dd"])
@pytest.mark.parametrize("types", [[D, D, D, D], [D, N, N, D], [N, D, D, N], [P, P, D, D], [D, N, P, P]])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_held_levels_have_the_oracles_bits(M, kind, nx, ny, types):
    v = Box.of_size(nx, ny)
    geo = G.mapped_geometry(v, G.map_skew_stretch(15.0, 1.02, 0.25, ny) if P not in types else G.map_identity())
    rng = np.random.default_rng(nx * 100 + ny)
    rhs = BoxData(v)
    rhs.data[:] = rng.standard_normal(rhs.data.shape)
    bc = BdryData(v, types, [BCMODE_UNIFORM] * 4)
    dd = kind == "dd"
    O.lib().or_set_dirichlet_coupled_diagonal.argtypes = [ctypes.c_int]
    O.lib().or_set_dirichlet_coupled_diagonal(1)
    po, pd = BoxData(v, 1, 1), BoxData(v, 1, 1)
    try:
        (O.dc_vcycle if dd else O.vcycle)(po, rhs.copy(), geo, bc, True, 1e-30, 2, numcycles=0, smooth_down=3,
                                          smooth_up=2, smooth_bottom=4, gs_order=1)
    finally:
        O.lib().or_set_dirichlet_coupled_diagonal(0)
    with M.Solver(v, geo, bc, KIND_DD if dd else KIND_MG, M.FLAG_DIRICHLET_COUPLED_DIAG) as s:
        (s.dc_vcycle if dd else s.vcycle)(pd, rhs.copy(), bc, True, 1e-30, 2, 0, 3, 2, 4)
    assert np.array_equal(po.interior(), pd.interior())
