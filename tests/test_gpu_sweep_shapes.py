"""The sweep kernel's shapes at their edges (csrc/mgp_sweep.cu), through a solver
that makes no coarse visit (numcycles = 0): per iteration eight sweeps, the
residual's restriction, the prolonged coarse guess and eight sweeps -- no
reduction enters the correction, so in FP64 every bit must be the oracle's in
the device's sweep order.  The sizes take each path: a level inside one window,
several sweeps a launch over tiles with remainders, one sweep a launch over the
large shape's frame and inner tiles, and its partition for a grid too narrow for
a frame."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from helpers import D, N, P, rand_geo
from mgpoisson2d_b200.types import BCMODE_UNIFORM, KIND_MG, BdryData, Box, BoxData
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# one window; 2 or 4 sweeps a launch; one sweep of small tiles; large tiles (frame of bands), exact multiples and remainders
SIZES = [(64, 48), (64, 56), (66, 58), (130, 94), (256, 256), (402, 390), (448, 416), (1700, 58), (58, 1700), (760, 110)]


@pytest.fixture(scope="module")
def M():
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as api
    return api


def _problem(nx, ny, types, seed=3):
    rng = np.random.default_rng(seed)
    v = Box.of_size(nx, ny)
    geo = rand_geo(v, rng)
    rhs = BoxData(v)
    rhs.data[:] = rng.standard_normal(rhs.data.shape)
    return v, geo, rhs, BdryData(v, types, [BCMODE_UNIFORM] * 4)


def _device(M, v, geo, rhs, bc, flags, nd, nu):
    phi = BoxData(v, 1, 1)
    with M.Solver(v, geo, bc, KIND_MG, flags, maxdepth_user=1) as s:
        rep = s.vcycle(phi, rhs, bc, True, 1e-30, 1, 0, nd, nu, 8)
    assert not rep.diverged   # else the correction would have been undone
    return phi.interior()


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("types", [[D, D, D, D], [D, D, N, N], [N, D, D, N], [P, P, D, D], [D, N, P, P]])
def test_sweeps_have_the_oracles_bits(M, nx, ny, types):
    v, geo, rhs, bc = _problem(nx, ny, types)
    O.lib().or_set_dirichlet_coupled_diagonal.argtypes = [ctypes.c_int]
    O.lib().or_set_dirichlet_coupled_diagonal(1)
    try:
        po = BoxData(v, 1, 1)
        O.vcycle(po, rhs, geo, bc, True, 1e-30, 1, maxdepth_user=1, numcycles=0, gs_order=1)
    finally:
        O.lib().or_set_dirichlet_coupled_diagonal(0)
    got = _device(M, v, geo, rhs, bc, M.FLAG_DIRICHLET_COUPLED_DIAG, 8, 8)
    assert np.array_equal(po.interior().view(np.uint64), np.ascontiguousarray(got).view(np.uint64).reshape(got.shape))


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("types", [[D, D, D, D], [N, D, D, N]])
def test_fp32_sweeps_follow_the_fp64_ones(M, nx, ny, types):
    """The same pass with FP32 grid levels.  16 sweeps of about 40 roundings of 2^-24, each relative to the largest
    value a sweep handles: 16 * 40 * 2^-24 = 4e-5 of the largest correction, doubled for the transfers."""
    v, geo, rhs, bc = _problem(nx, ny, types)
    a = _device(M, v, geo, rhs, bc, M.FLAG_DIRICHLET_COUPLED_DIAG, 8, 8)
    b = _device(M, v, geo, rhs, bc, M.FLAG_DIRICHLET_COUPLED_DIAG | M.FLAG_MIXED, 8, 8)
    assert np.abs(a - b).max() <= 8e-5 * np.abs(a).max()


@pytest.mark.parametrize("nd,nu", [(1, 3), (2, 5), (6, 7)])
@pytest.mark.parametrize("mixed", [False, True])
def test_counts_that_no_launch_size_divides(M, nd, nu, mixed):
    """nd and nu split into launches of 4, 2 and 1 sweeps (bounds as above)."""
    nx, ny = 130, 94
    v, geo, rhs, bc = _problem(nx, ny, [D, D, N, N])
    O.lib().or_set_dirichlet_coupled_diagonal.argtypes = [ctypes.c_int]
    O.lib().or_set_dirichlet_coupled_diagonal(1)
    try:
        po = BoxData(v, 1, 1)
        O.vcycle(po, rhs, geo, bc, True, 1e-30, 1, maxdepth_user=1, numcycles=0, smooth_down=nd, smooth_up=nu,
                 gs_order=1)
    finally:
        O.lib().or_set_dirichlet_coupled_diagonal(0)
    flags = M.FLAG_DIRICHLET_COUPLED_DIAG | (M.FLAG_MIXED if mixed else 0)
    got = _device(M, v, geo, rhs, bc, flags, nd, nu)
    want = po.interior()
    if mixed:
        assert np.abs(got - want).max() <= 8e-5 * np.abs(want).max()
    else:
        assert np.array_equal(np.ascontiguousarray(got), np.ascontiguousarray(want))
