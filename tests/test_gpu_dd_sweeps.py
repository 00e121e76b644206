"""Several red-black sweeps of the deferred-correction smoother in one launch
(csrc/mgp_ddsweep.cu): one V-cycle without a coarse visit (numcycles = 0), where no
reduction enters the correction, so in FP64 every bit of phi -- ghosts the next
residual reads included -- must be the oracle's.  Sizes: one window, tiles with
remainders, more tiles than SMs, thin grids; counts that 4 and 2 do not divide."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import D, N, P, rand_geo
from mgpoisson2d_b200.types import BCMODE_UNIFORM, KIND_DD, BdryData, Box, BoxData
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SIZES = [(64, 32), (64, 64), (66, 34), (130, 94), (256, 256), (602, 390), (1700, 38), (38, 1700)]


@pytest.fixture(scope="module")
def M():
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as api
    return api


def _problem(nx, ny, types):
    rng = np.random.default_rng(5)
    v = Box.of_size(nx, ny)
    geo = rand_geo(v, rng, cross=0.1)
    rhs = BoxData(v)
    rhs.data[:] = rng.standard_normal(rhs.data.shape)
    return v, geo, rhs, BdryData(v, types, [BCMODE_UNIFORM] * 4)


def _device(M, v, geo, rhs, bc, flags, nd, nu):
    phi = BoxData(v, 1, 1)
    with M.Solver(v, geo, bc, KIND_DD, flags, maxdepth_user=1) as s:
        rep = s.dc_vcycle(phi, rhs.copy(), bc, True, 1e-30, 1, 0, nd, nu, 8)
    assert not rep.diverged   # else the correction would have been undone
    return phi.interior()


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("types", [[D, D, D, D], [N, D, D, N], [D, D, N, N], [P, P, D, D]])
@pytest.mark.parametrize("nd,nu", [(8, 8), (1, 3), (5, 6)])
def test_dd_sweeps_follow_the_oracle(M, nx, ny, types, nd, nu):
    v, geo, rhs, bc = _problem(nx, ny, types)
    po = BoxData(v, 1, 1)
    O.dc_vcycle(po, rhs.copy(), geo, bc, True, 1e-30, 1, maxdepth_user=1, numcycles=0, smooth_down=nd, smooth_up=nu,
                gs_order=1)
    want = np.ascontiguousarray(po.interior())
    a = np.ascontiguousarray(_device(M, v, geo, rhs, bc, 0, nd, nu))
    assert np.array_equal(want.view(np.uint64), a.view(np.uint64))
    # FP32 grid levels: nd + nu sweeps of about 25 roundings of 2^-24 each, relative to the largest value a sweep handles,
    # doubled for the transfers
    b = _device(M, v, geo, rhs, bc, M.FLAG_MIXED, nd, nu)
    assert np.abs(a - b).max() <= 2 * (nd + nu) * 25 * 2.0 ** -24 * np.abs(a).max()
