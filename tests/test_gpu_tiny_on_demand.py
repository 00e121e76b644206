"""Under the exact bottom of the coarse-cycle level (MGP_FLAG_DIRECT_LARGE) a V-cycle never
goes below it: the dense forms of the levels there are made when fmg first starts on them,
not with every solver."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import D, rand_field
from mgpoisson2d_b200 import geometry as G
from mgpoisson2d_b200.types import BCMODE_UNIFORM, KIND_MG, BdryData, Box, BoxData

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_fmg_makes_the_dense_forms_once():
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as M

    v = Box.of_size(32, 32)
    geo = G.mapped_geometry(v, G.map_skew_stretch(10.0, 1.02, 0.25, 32))
    rhs = rand_field(v, np.random.default_rng(1), 0)
    bc = BdryData(v, [D] * 4, [BCMODE_UNIFORM] * 4)
    flags = M.FLAG_DIRICHLET_COUPLED_DIAG | M.FLAG_DIRECT_COARSE | M.FLAG_DIRECT_LARGE
    with M.Solver(v, geo, bc, KIND_MG, flags) as s:
        def launches(call):
            phi = BoxData(v, 1, 1)
            n0 = M.kernel_launch_count()
            r = call(phi, rhs, bc, True, 1e-10, 5)
            assert r.final_relres <= 1e-10
            return M.kernel_launch_count() - n0, phi.interior().copy()
        launches(s.vcycle)
        a, pa = launches(s.fmg)
        b, pb = launches(s.fmg)
    assert a - b == 2   # a launch for 8 x 8 and for 4 x 4
    assert np.array_equal(pa, pb)
