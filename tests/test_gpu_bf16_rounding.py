"""MGP_FLAG_BF16_COARSE rounds the correction of a level after two sweeps where 32 x 32
tiles are at most two an SM and no side is periodic, else after each sweep -- however many
sweeps the launches make.  The residual after one V-cycle shows which: it was measured when
two sweeps always shared a launch on such levels.  Values that fall to the other side of a
rounding boundary (the FP32 sweeps' own rounding decides) move it by a few thousandths, a
rounding more per two sweeps by a quarter; 5 % lies between."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import D, P
from mgpoisson2d_b200 import geometry as G
from mgpoisson2d_b200.types import BCMODE_UNIFORM, KIND_MG, BdryData, Box, BoxData

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def M():
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as api
    return api


@pytest.mark.parametrize("nx,ny,types,nd,nu,relres", [
    (1024, 512, [D] * 4, 8, 8, 6.411e-3),          # level 1: 128 tiles, more windows of two sweeps than fit a wave
    (1024, 1024, [D] * 4, 8, 8, 7.784e-3),         # 256 tiles
    (1280, 896, [D] * 4, 3, 5, 1.983e-2),          # odd counts: the last sweep is rounded by itself
    (1024, 1024, [P, P, D, D], 8, 8, 1.0958e-2)])  # a periodic side: after each sweep
def test_rounds_as_often_as_it_says(M, nx, ny, types, nd, nu, relres):
    v = Box.of_size(nx, ny)
    geo = G.mapped_geometry(v, G.map_identity())
    rhs = BoxData(v)
    rhs.data[:] = np.random.default_rng(7).standard_normal(rhs.data.shape)
    bc = BdryData(v, types, [BCMODE_UNIFORM] * 4)
    flags = M.FLAG_MIXED | M.FLAG_BF16_COARSE | M.FLAG_DIRICHLET_COUPLED_DIAG
    with M.Solver(v, geo, bc, KIND_MG, flags) as s:
        r = s.vcycle(BoxData(v, 1, 1), rhs, bc, True, 1e-30, 1, 1, nd, nu, 8)
    assert r.relres[1] == pytest.approx(relres, rel=0.05)
