"""Bottoms of up to 3600 cells that no CTA stages and no window holds run the general phases
in CTAs of 256 threads (k_coarse_jobs_plain, k_bicgstab_plain): a lockstep batch of them
beside staged and larger ones has the bits of each problem alone, and the operator-level
solve_bicgstab2 follows the oracle at the edges of its rule."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import D, N, P, rand_field
from mgpoisson2d_b200 import geometry as G
from mgpoisson2d_b200.types import BCMODE_UNIFORM, KIND_MG, BdryData, Box, BoxData
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
    geo = G.mapped_geometry(v, G.map_identity() if P in types else G.map_skew_stretch(15.0, 1.02, 0.25, ny))
    return v, geo, rand_field(v, np.random.default_rng(nx * 1000 + ny), 0), BdryData(v, types, [BCMODE_UNIFORM] * 4)


# bottoms: 59 x 61 and 75 x 48 (3599 and 3600 cells) are the last plain ones, 61 x 61 is past them, 33 x 33 is staged
@pytest.mark.parametrize("sizes", [[(59, 61)], [(51, 53), (49, 51)], [(59, 61), (33, 33), (64, 64)],
                                   [(102, 106), (75, 48), (61, 61), (74, 66), (130, 122)]])
@pytest.mark.parametrize("types", [[D, D, D, D], [D, N, N, D]])
def test_a_lockstep_batch_has_the_bits_of_each_alone(M, sizes, types):
    probs = [_problem(nx, ny, types) for nx, ny in sizes]
    flags = M.FLAG_DIRICHLET_COUPLED_DIAG
    with M.Batch([(v, g, bc) for v, g, _, bc in probs], KIND_MG, flags | M.FLAG_LOCKSTEP) as b:
        b.set_tuning(1, 0)
        phis = [BoxData(p[0], 1, 1) for p in probs]
        b.vcycle(phis, [p[2] for p in probs], [p[3] for p in probs], True, 1e-30, 3)
    for (v, geo, rhs, bc), got in zip(probs, phis):
        with M.Solver(v, geo, bc, KIND_MG, flags) as s:
            phi = BoxData(v, 1, 1)
            s.vcycle(phi, rhs, bc, True, 1e-30, 3)
        assert np.array_equal(phi.interior(), got.interior()) and np.abs(phi.interior()).max() > 0


@pytest.mark.parametrize("types", [[D, D, D, D], [D, N, N, D], [P, P, D, D], [D, D, P, P]])
@pytest.mark.parametrize("nx,ny", [(4, 16), (8, 8), (13, 5), (16, 16), (53, 25), (60, 60), (61, 59), (61, 60)])
def test_bicgstab_follows_the_oracle(M, nx, ny, types):
    v, geo, rhs, bc = _problem(nx, ny, types)
    a, b, inv = BoxData(v, 1, 1), BoxData(v, 1, 1), BoxData(v)
    O.compute_invdiags(inv, geo, bc, True)
    O.solve_bicgstab2(a, rhs, geo, bc, True, inv, 1e-30, 2, 0, False, 0, gs_order=1)
    M.solve_bicgstab2(b, rhs, geo, bc, True, inv, 1e-30, 2, 0, False, 0)
    # sums of up to 3660 terms in another order: 4e-13 in each of some ten scalars of two iterations
    assert np.abs(a.interior()).max() > 0
    assert np.abs(a.interior() - b.interior()).max() <= 1e-10 * np.abs(a.interior()).max()
