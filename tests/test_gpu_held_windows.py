"""The windows in which one CTA sweeps a nine-point level it holds (mgp_sweep.cuh: 32 x 48,
64 x 24, 40 x 38, 48 x 32 and 52 x 28 cells; the general phases beyond): at their edges and
one past them.  Two BiCGStab iterations, eight preconditioner sweeps, follow the oracle's, and sizes
that a coarse level of at most 1024 cells can have keep its bits through the sweeps alone."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from helpers import D, N, P, rand_bc, rand_field
from mgpoisson2d_b200 import geometry as G
from mgpoisson2d_b200.types import BCMODE_NONUNIFORM, BCMODE_UNIFORM, KIND_MG, BdryData, Box, BoxData
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def M():
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as api
    return api


def _geo(v, types):
    return G.mapped_geometry(v, G.map_identity() if P in types else G.map_skew_stretch(15.0, 1.02, 0.25, v.ny))


@pytest.mark.parametrize("types", [[D, D, D, D], [D, N, N, D], [N, D, D, N], [P, P, D, D], [D, N, P, P]])
@pytest.mark.parametrize("nx,ny", [(32, 48), (33, 33), (40, 38), (39, 38), (40, 37), (41, 25), (48, 32), (47, 31),
                                   (49, 28), (52, 27), (52, 28), (53, 24), (64, 24), (33, 39), (41, 33), (53, 25)])
def test_bicgstab_iterations_follow_the_oracle(M, nx, ny, types):
    v = Box.of_size(nx, ny)
    geo = _geo(v, types)
    rng = np.random.default_rng(nx * 100 + ny)
    homog = P in types
    bc = rand_bc(v, types, [BCMODE_UNIFORM, BCMODE_NONUNIFORM, BCMODE_UNIFORM, BCMODE_UNIFORM] if not homog
                 else [BCMODE_UNIFORM] * 4, rng)
    rhs, a = rand_field(v, rng, 0), rand_field(v, rng, 1)
    b, inv = a.copy(), BoxData(v)
    O.compute_invdiags(inv, geo, bc, homog)
    O.solve_bicgstab2(a, rhs, geo, bc, homog, inv, 1e-30, 2, 0, False, 0, gs_order=1)
    M.solve_bicgstab2(b, rhs, geo, bc, homog, inv, 1e-30, 2, 0, False, 0)
    # sums of up to 2000 terms in another order: 2000 * 2^-53 = 2e-13 in each of some ten scalars of two iterations
    assert np.isfinite(a.interior()).all() and np.abs(a.interior()).max() > 0
    assert np.abs(a.interior() - b.interior()).max() <= 1e-10 * np.abs(a.interior()).max()


@pytest.mark.parametrize("types", [[D, D, D, D], [D, N, N, D], [N, D, D, N], [P, P, D, D], [D, N, P, P]])
@pytest.mark.parametrize("nx,ny", [(34, 30), (36, 28), (38, 26), (16, 48), (40, 24)])
def test_levels_keep_the_oracles_bits(M, nx, ny, types):
    v = Box.of_size(nx, ny)
    geo, rhs = _geo(v, types), BoxData(v)
    # a smooth right-hand side: the sweeps and the guess of the level below lower its residual, so the cycle is kept
    x, y = np.meshgrid((np.arange(nx) + 0.5) / nx, (np.arange(ny) + 0.5) / ny, indexing="ij")
    rhs.data[:] = np.sin(5 * np.pi * x) * np.sin(7 * np.pi * y) + 0.1 * np.random.default_rng(nx).standard_normal((nx, ny))
    bc = BdryData(v, types, [BCMODE_UNIFORM] * 4)
    O.lib().or_set_dirichlet_coupled_diagonal.argtypes = [ctypes.c_int]
    O.lib().or_set_dirichlet_coupled_diagonal(1)
    po, pd = BoxData(v, 1, 1), BoxData(v, 1, 1)
    try:
        ro = O.vcycle(po, rhs.copy(), geo, bc, True, 1e-30, 2, numcycles=0, smooth_down=3, smooth_up=2,
                      smooth_bottom=4, gs_order=1)
    finally:
        O.lib().or_set_dirichlet_coupled_diagonal(0)
    with M.Solver(v, geo, bc, KIND_MG, M.FLAG_DIRICHLET_COUPLED_DIAG) as s:
        rd = s.vcycle(pd, rhs.copy(), bc, True, 1e-30, 2, 0, 3, 2, 4)
    assert rd.iterations == ro.iterations and rd.iterations > 0 and not rd.diverged and not ro.diverged
    assert np.abs(po.interior()).max() > 0
    assert np.array_equal(po.interior(), pd.interior())
