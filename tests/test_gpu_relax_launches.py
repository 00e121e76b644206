"""Launches of relax_gs on a caller's arrays that outnumber the SMs in tiles
(sweep_plan, csrc/mgp_sweep.cu): pairs of sweeps up to six rounds of their tiles, one
sweep a launch above, and the same bits either way as sweep by sweep."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import D, N, rand_field, rand_geo, same
from mgpoisson2d_b200.types import BCMODE_UNIFORM, BdryData, Box

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nx,ny,launches", [(450, 448, 4), (901, 700, 8)])
def test_eight_sweeps(nx, ny, launches):
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as M

    rng = np.random.default_rng(nx)
    v = Box.of_size(nx, ny)
    geo, rhs, inv = rand_geo(v, rng).to_device(), rand_field(v, rng, 0).to_device(), rand_field(v, rng, 0)
    inv.data[:] = -1e-7 * (1.0 + 0.1 * inv.data)
    inv, start = inv.to_device(), rand_field(v, rng)
    bc = BdryData(v, [D, N, D, D], [BCMODE_UNIFORM] * 4)

    def sweeps(counts):
        phi = start.to_device()
        n0 = M.kernel_launch_count()
        for n in counts:
            M.relax_gs(phi, rhs, geo, bc, True, inv, 1.0, -1.0, n, False)
        return phi, M.kernel_launch_count() - n0
    one, n1 = sweeps([8])
    two, n2 = sweeps([1] * 8)
    assert same(np.ascontiguousarray(one.host()), np.ascontiguousarray(two.host()))
    assert n1 == launches and n2 == 8
