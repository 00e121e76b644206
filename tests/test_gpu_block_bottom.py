"""The exact bottom of more than 1024 cells (csrc/mgp_bottom.cu): a grid that does
not coarsen is its own bottom, so one V-cycle without smoothing above it is the
exact solve: the oracle forms its residual.  Odd and even
line counts (the first step of the reduction differs), lines along either axis, a
periodic side either way, block sizes on both sides of a warp's multiple; and a
level beyond the largest line, which keeps the reference bottom."""
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
    geo = G.mapped_geometry(v, G.map_skew_stretch(15.0, 1.02, 0.25, ny) if P not in types else G.map_identity())
    rng = np.random.default_rng(nx * 1000 + ny)
    return v, geo, rand_field(v, rng, 0), BdryData(v, types, [BCMODE_UNIFORM] * 4)


DDDD, DNND, PPDD, DDPP = [D, D, D, D], [D, N, N, D], [P, P, D, D], [D, D, P, P]


@pytest.mark.parametrize("nx,ny,types", [
    (33, 33, DDDD), (35, 31, DNND), (31, 36, DNND), (37, 31, PPDD), (29, 39, DDPP), (5, 211, DDDD), (206, 5, DNND),
    (33, 32, PPDD), (65, 33, DDDD)])
def test_exact_bottom_is_the_solution(M, nx, ny, types):
    v, geo, rhs, bc = _problem(nx, ny, types)
    flags = M.FLAG_DIRICHLET_COUPLED_DIAG | M.FLAG_DIRECT_COARSE | M.FLAG_DIRECT_LARGE
    n0 = M.kernel_launch_count()
    with M.Solver(v, geo, bc, KIND_MG, flags) as s:
        phi = BoxData(v, 1, 1)
        r = s.vcycle(phi, rhs, bc, True, 1e-10, 5)
        phi2 = BoxData(v, 1, 1)
        s.vcycle(phi2, rhs, bc, True, 1e-10, 5)
    assert M.kernel_launch_count() > n0
    assert r.status == 0 and r.iterations == 1 and r.final_relres <= 1e-10, (r.iterations, r.final_relres)
    assert np.array_equal(phi.interior(), phi2.interior())
    # the residual bounds the error by the operator's condition; the oracle forms it on its own
    res = BoxData(v)
    O.compute_residual(res, rhs, phi.copy(), geo, bc, True)
    assert np.linalg.norm(res.interior()) <= 1e-10 * np.linalg.norm(rhs.interior())


def test_beyond_the_largest_line_the_reference_bottom_stays(M):
    v, geo, rhs, bc = _problem(163, 161, DDDD)
    base = M.FLAG_DIRICHLET_COUPLED_DIAG | M.FLAG_DIRECT_COARSE
    sols = []
    for flags in (base, base | M.FLAG_DIRECT_LARGE):
        with M.Solver(v, geo, bc, KIND_MG, flags) as s:
            phi = BoxData(v, 1, 1)
            s.vcycle(phi, rhs, bc, True, 1e-6, 1)
        sols.append(phi.interior().copy())
    assert np.array_equal(sols[0], sols[1])


def test_gmres_above_an_exact_bottom_of_many_cells(M):
    """105 x 54 below two coarsenings: GMRES with the exact bottom takes no more
    V-cycles than with the reference bottom (which stops at 1e-6) and reaches the
    same solution."""
    v, geo, rhs, bc = _problem(420, 216, DDDD)
    base = M.FLAG_DIRICHLET_COUPLED_DIAG | M.FLAG_GMRES | M.FLAG_DIRECT_COARSE
    out = []
    for flags in (base, base | M.FLAG_DIRECT_LARGE, base | M.FLAG_DIRECT_LARGE | M.FLAG_MIXED):
        with M.Solver(v, geo, bc, KIND_MG, flags) as s:
            phi = BoxData(v, 1, 1)
            r = s.vcycle(phi, rhs, bc, True, 1e-10, 100)
        assert r.status == 0 and r.final_relres <= 1e-10
        out.append((r.iterations, phi.interior().copy()))
    scale = np.abs(out[0][1]).max()
    for it, p in out[1:]:
        assert it <= out[0][0] + 1
        assert np.abs(p - out[0][1]).max() <= 1e-7 * scale


def test_lockstep_over_exact_bottoms_has_the_bits_of_each_alone(M):
    probs = [_problem(nx, ny, DDDD) for nx, ny in ((140, 132), (74, 66), (64, 64))]
    flags = M.FLAG_DIRICHLET_COUPLED_DIAG | M.FLAG_DIRECT_COARSE | M.FLAG_DIRECT_LARGE
    with M.Batch([(v, g, bc) for v, g, _, bc in probs], KIND_MG, flags | M.FLAG_LOCKSTEP) as b:
        phis = [BoxData(p[0], 1, 1) for p in probs]
        b.vcycle(phis, [p[2] for p in probs], [p[3] for p in probs], True, 1e-9, 60)
    for (v, geo, rhs, bc), got in zip(probs, phis):
        with M.Solver(v, geo, bc, KIND_MG, flags) as s:
            phi = BoxData(v, 1, 1)
            s.vcycle(phi, rhs, bc, True, 1e-9, 60)
        assert np.array_equal(phi.interior(), got.interior())
