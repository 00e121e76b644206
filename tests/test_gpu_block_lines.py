"""The exact bottom of more than 1024 cells (csrc/mgp_bottom.cu) over the rest of its range:
lines of 55 to 160 cells (blocks of more than 48 KB of shared memory from 79 on, every
32-column share of a row), the most lines, the launches of a solve; and the levels that keep
the reference bottom, because the factors would take more than 256 MB or do not solve."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import D, N, P, rand_field
from mgpoisson2d_b200 import geometry as G
from mgpoisson2d_b200.types import BCMODE_UNIFORM, KIND_MG, BdryData, Box, BoxData
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

DDDD, DNND, PPDD, NNNN = [D, D, D, D], [D, N, N, D], [P, P, D, D], [N, N, N, N]


@pytest.fixture(scope="module")
def M():
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as api
    return api


def _problem(nx, ny, types):
    plain = P in types or max(nx, ny) > 1000
    v = Box.of_size(nx, ny, 1.0, ny / nx if plain else 1.0)   # (the plain ones of square cells)
    geo = G.mapped_geometry(v, G.map_identity() if plain else G.map_skew_stretch(15.0, 1.01, 0.25, ny))
    rhs = rand_field(v, np.random.default_rng(nx * 1000 + ny), 0)
    if D not in types:
        rhs.data -= rhs.data.mean()
    return v, geo, rhs, BdryData(v, types, [BCMODE_UNIFORM] * 4)


def _flags(M):
    return M.FLAG_DIRICHLET_COUPLED_DIAG | M.FLAG_DIRECT_COARSE


def _steps(lines):
    n, first, steps = lines, True, 0
    while n > 1:
        n = n // 2 + 1 if first and n % 2 == 0 else (n + 1) // 2
        first = False
        steps += 1
    return steps


@pytest.mark.parametrize("nx,ny,types", [
    (55, 64, DNND), (65, 66, PPDD), (78, 81, DDDD), (79, 80, DNND), (83, 79, DDDD), (96, 97, DDDD), (97, 129, DNND),
    (131, 128, PPDD), (129, 131, DDDD), (159, 163, DNND), (160, 161, DDDD), (5, 16384, DDDD)])
def test_solves_over_its_range(M, nx, ny, types):
    v, geo, rhs, bc = _problem(nx, ny, types)
    launches = []
    for flags in (_flags(M), _flags(M) | M.FLAG_DIRECT_LARGE):
        with M.Solver(v, geo, bc, KIND_MG, flags) as s:
            phi = BoxData(v, 1, 1)
            n0 = M.kernel_launch_count()
            r = s.vcycle(phi, rhs, bc, True, 1e-300, 1)
            launches.append(M.kernel_launch_count() - n0)
    # the grid is its own bottom: BiCGStab is one launch, the reduction one a step down and up and one between
    assert launches[1] - launches[0] == 2 * _steps(ny if P in types else max(nx, ny))
    assert r.status == 0 and r.iterations == 1 and not r.diverged
    res = BoxData(v)
    O.compute_residual(res, rhs, phi.copy(), geo, bc, True)
    assert np.linalg.norm(res.interior()) <= 1e-10 * np.linalg.norm(rhs.interior())


@pytest.mark.parametrize("nx,ny,types", [(160, 263, DDDD),   # 269 MB of factors
                                         (5, 16385, DDDD),   # more lines than a launch has products for
                                         (33, 35, NNNN), (64, 71, NNNN)])   # singular: the factors are tried and rejected
def test_keeps_the_reference_bottom(M, nx, ny, types):
    v, geo, rhs, bc = _problem(nx, ny, types)
    out = []
    for flags in (_flags(M), _flags(M) | M.FLAG_DIRECT_LARGE):
        with M.Solver(v, geo, bc, KIND_MG, flags) as s:
            phi = BoxData(v, 1, 1)
            n0 = M.kernel_launch_count()
            s.vcycle(phi, rhs, bc, True, 1e-6, 1)
            out.append((M.kernel_launch_count() - n0, phi.interior().copy()))
    assert out[0][0] == out[1][0]
    assert np.abs(out[0][1]).max() > 0
    assert np.array_equal(out[0][1], out[1][1])
