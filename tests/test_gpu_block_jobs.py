"""Exact bottoms of more than 1024 cells in a lockstep batch: the steps of all problems'
reductions share launches (k_bb_jobs, csrc/mgp_bottom.cu), whatever their sizes, numbers
of lines and direction, and each problem keeps the bits it has alone."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import D, N, rand_field
from mgpoisson2d_b200 import geometry as G
from mgpoisson2d_b200.types import BCMODE_UNIFORM, KIND_MG, BdryData, Box, BoxData

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def M():
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as api
    return api


def _problem(nx, ny, types=(D, D, D, D)):
    v = Box.of_size(nx, ny)
    geo = G.mapped_geometry(v, G.map_skew_stretch(15.0, 1.02, 0.25, ny))
    rng = np.random.default_rng(nx * 1000 + ny)
    return v, geo, rand_field(v, rng, 0), BdryData(v, list(types), [BCMODE_UNIFORM] * 4)


def _flags(M):
    return M.FLAG_DIRICHLET_COUPLED_DIAG | M.FLAG_DIRECT_COARSE | M.FLAG_DIRECT_LARGE


# bottoms 33 x 35, 7 x 211 and 211 x 7 (longest reduction first and last), 35 x 37; 16 x 16 has a dense one
@pytest.mark.parametrize("mixed", [False, True])
def test_problems_of_unequal_steps_have_the_bits_of_each_alone(M, mixed):
    probs = [_problem(66, 70), _problem(14, 422), _problem(422, 14, (D, N, N, D)), _problem(140, 148), _problem(64, 64)]
    flags = _flags(M) | (M.FLAG_MIXED if mixed else 0)
    for order in (probs, probs[::-1]):
        with M.Batch([(v, g, bc) for v, g, _, bc in order], KIND_MG, flags | M.FLAG_LOCKSTEP, nstreams=1) as b:
            phis = [BoxData(p[0], 1, 1) for p in order]
            reps = b.vcycle(phis, [p[2] for p in order], [p[3] for p in order], True, 1e-8, 40)
        for (v, geo, rhs, bc), got, rep in zip(order, phis, reps):
            with M.Solver(v, geo, bc, KIND_MG, flags) as s:
                phi = BoxData(v, 1, 1)
                r = s.vcycle(phi, rhs, bc, True, 1e-8, 40)
            assert r.iterations == rep.iterations and not r.diverged
            assert np.array_equal(phi.interior(), got.interior())


def test_more_problems_take_no_more_launches(M):
    counts = []
    for n in (2, 9):
        probs = [_problem(66, 70)] * n
        with M.Batch([(v, g, bc) for v, g, _, bc in probs], KIND_MG, _flags(M) | M.FLAG_LOCKSTEP, nstreams=1) as b:
            phis = [BoxData(p[0], 1, 1) for p in probs]
            n0 = M.kernel_launch_count()
            b.vcycle(phis, [p[2] for p in probs], [p[3] for p in probs], True, 1e-30, 3)
            counts.append(M.kernel_launch_count() - n0)
    assert counts[0] == counts[1], counts
