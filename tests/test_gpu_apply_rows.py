"""The operator kernel walks two cells up a column: heights and widths at which a
thread's second cell is missing, on a side, or the only interior one, in every
kind of side, bit for bit as the oracle computes them."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import D, N, P, rand_bc, rand_field, rand_geo, same
from mgpoisson2d_b200.types import BCMODE_NONUNIFORM, BCMODE_UNIFORM, Box
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("types", [[D, N, N, D], [P, P, P, P]], ids=["sides", "periodic"])
@pytest.mark.parametrize("nx,ny", [(3, 3), (4, 5), (33, 4), (32, 17), (65, 16), (31, 18), (34, 33)])
def test_operator_at_row_remainders(nx, ny, types):
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as M

    rng = np.random.default_rng(nx * 64 + ny)
    v = Box.of_size(nx, ny)
    geo, phi, rhs = rand_geo(v, rng), rand_field(v, rng), rand_field(v, rng, 0)
    u, n = BCMODE_UNIFORM, BCMODE_NONUNIFORM
    bc = rand_bc(v, types, [u] * 4 if P in types else [n, u, u, n], rng)
    lap_o, res_o, phi_o = rand_field(v, rng, 0), rand_field(v, rng, 0), phi.copy()
    lap, res, phi_d = lap_o.copy(), res_o.copy(), phi.copy()
    O.compute_laplacian(lap_o, phi_o, geo, bc, False)
    M.compute_laplacian(lap, phi_d, geo, bc, False)
    assert same(lap.data, lap_o.data)
    O.compute_residual(res_o, rhs, phi_o, geo, bc, True)
    M.compute_residual(res, rhs, phi_d, geo, bc, True)
    assert same(res.data, res_o.data) and same(phi_d.data, phi_o.data)
