"""The first sweep's ghosts of sides that the window's rows do not give (start_ghosts,
csrc/mgp_sweep.cuh): read from phi as it stands before the launch, beside the window's own
loads.  Doubly periodic grids, whose corner ghosts are cells of the far corner, at the edges
of each shape; and inhomogeneous sides, whose later ghosts in the same launch come from the
window."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import D, N, NU, P, U, rand_bc, rand_field, rand_geo, same
from mgpoisson2d_b200.types import KIND_MG, BCMODE_UNIFORM, BdryData, Box, BoxData
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def M():
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as api
    return api


# a window, one cell more either way, tiles with remainders, more than a round of them
@pytest.mark.parametrize("nx,ny", [(4, 4), (32, 48), (33, 48), (32, 49), (45, 37), (130, 94), (402, 391)])
@pytest.mark.parametrize("types,modes", [([P, P, P, P], [U] * 4), ([P, P, D, N], [U, U, NU, U]), ([D, D, P, P], [NU, U, U, U]),
                                         ([D, N, D, D], [NU, U, U, NU])], ids=["PPPP", "PPDN", "DDPP", "DNDD"])
def test_sweeps_of_a_callers_arrays_have_the_oracles_bits(M, nx, ny, types, modes):
    rng = np.random.default_rng(nx * 7 + ny)
    v = Box.of_size(nx, ny)
    geo, rhs, phi, inv = rand_geo(v, rng), rand_field(v, rng, 0), rand_field(v, rng), rand_field(v, rng, 0)
    inv.data[:] = -1e-4 * (1.0 + 0.1 * inv.data)
    if NU in modes and v.jlo != v.ilo:
        pytest.skip("y-side values need jlo == ilo")
    bc = rand_bc(v, types, modes, rng)
    po, pd = phi.copy(), phi.copy()
    O.relax_gs(po, rhs, geo, bc, False, inv, 0.9, -1.0, 3, False, gs_order=1)
    M.relax_gs(pd, rhs, geo, bc, False, inv, 0.9, -1.0, 3, False)
    assert same(np.ascontiguousarray(po.data), np.ascontiguousarray(pd.data))


@pytest.mark.parametrize("nx,ny", [(64, 56), (130, 94), (402, 390), (1700, 58), (58, 1700)])
def test_doubly_periodic_levels_of_a_solver_follow_the_oracle(M, nx, ny):
    """One V-cycle without a coarse visit; the mean that its prolongation takes out of the correction is summed in another
    order: n roundings of 2^-53 of the largest value, doubled for the sweeps after it."""
    rng = np.random.default_rng(nx)
    v = Box.of_size(nx, ny)
    geo, rhs = rand_geo(v, rng), rand_field(v, rng, 0)
    bc = BdryData(v, [P] * 4, [BCMODE_UNIFORM] * 4)
    po, pd = BoxData(v, 1, 1), BoxData(v, 1, 1)
    O.vcycle(po, rhs, geo, bc, True, 1e-30, 1, maxdepth_user=1, numcycles=0, gs_order=1)
    with M.Solver(v, geo, bc, KIND_MG, 0, maxdepth_user=1) as s:
        rep = s.vcycle(pd, rhs, bc, True, 1e-30, 1, 0, 8, 8, 8)
    a, b = po.interior(), pd.interior()
    assert not rep.diverged and np.abs(a).max() > 0
    assert np.abs(a - b).max() <= 2 * nx * ny * 2.0 ** -53 * np.abs(a).max()
