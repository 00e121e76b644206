"""The server's memory budget and the optional factors of a large exact bottom
(MGP_FLAG_DIRECT_LARGE above 1024 cells): they count against the budget before they are
made, and a request whose hierarchy fits only without them is served, with the reference
bottom, as if the flag were not given."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import D, rand_field
from mgpoisson2d_b200 import geometry as G
from mgpoisson2d_b200.types import BCMODE_UNIFORM, KIND_MG, BdryData, Box, BoxData

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def M():
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as api
    return api


# 95 x 95 is its own bottom: some 10 MB estimated for the hierarchy, 51 MB more while 34 MB of factors are made
N = 95


def _problem():
    v = Box.of_size(N, N)
    geo = G.mapped_geometry(v, G.map_skew_stretch(15.0, 1.02, 0.25, N))
    return v, geo, rand_field(v, np.random.default_rng(N), 0), BdryData(v, [D] * 4, [BCMODE_UNIFORM] * 4)


@pytest.mark.parametrize("budget,exact", [(16 << 20, False), (48 << 20, False), (72 << 20, True)])
def test_factors_are_made_where_the_budget_holds_them(M, budget, exact):
    v, geo, rhs, bc = _problem()
    base = M.FLAG_DIRICHLET_COUPLED_DIAG | M.FLAG_DIRECT_COARSE
    want = BoxData(v, 1, 1)
    with M.Solver(v, geo, bc, KIND_MG, base | (M.FLAG_DIRECT_LARGE if exact else 0)) as s:
        s.vcycle(want, rhs, bc, True, 1e-10, 10, zerophi=True)
    with M.Server(2, budget, base | M.FLAG_DIRECT_LARGE) as srv:   # room for one at a time, on two workers
        phis = [BoxData(v, 1, 1) for _ in range(3)]
        tickets = [srv.submit(v, geo, bc, p, rhs, True, 1e-10, 10, zerophi=True) for p in phis]
        reps = [srv.wait(t)[0] for t in tickets]
    for r, p in zip(reps, phis):
        assert r.final_relres <= 1e-10
        assert np.array_equal(p.interior(), want.interior())
