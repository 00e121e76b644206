"""Operator-level calls work on device arrays where they lie; host arrays, arrays
without the ghosts a kernel needs and arrays that share memory are staged.  Every
call must give the same bits either way, whatever shares memory with what."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import D, N, rand_bc, rand_field, rand_geo, same
from mgpoisson2d_b200.types import BCMODE_NONUNIFORM, BCMODE_UNIFORM, BD_CELL, BD_NODE, Box, BoxData, GeoData

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

NX, NY = 37, 29


@pytest.fixture(scope="module")
def M():
    assert torch.cuda.is_available(), "needs a CUDA device"
    import mgpoisson2d_b200.api as api
    return api


class World:
    """The arrays of the calls below, on the host or on the device."""

    def __init__(self, device: bool):
        rng = np.random.default_rng(8)
        v = self.v = Box.of_size(NX, NY)
        u, nu = BCMODE_UNIFORM, BCMODE_NONUNIFORM
        self.bc = rand_bc(v, [D, N, D, D], [u, nu, nu, u], rng)
        geo = rand_geo(v, rng)
        self.phi, self.rhs, self.out = rand_field(v, rng), rand_field(v, rng, 0), rand_field(v, rng, 0)
        self.bare = rand_field(v, rng, 0)   # phi without ghosts
        self.inv = rand_field(v, rng, 0)
        self.inv.data[:] = -1e-4 * (1.0 + 0.1 * self.inv.data)
        self.xf, self.yf = rand_field(v, rng, 0, BD_NODE, BD_CELL), rand_field(v, rng, 1, BD_CELL, BD_NODE)
        f = self.fv = Box.of_size(2 * 24, 2 * 18)
        c = self.cv = f.coarsened(2, 2)
        self.fine, self.crse = rand_field(f, rng, 2), rand_field(c, rng, 1)
        self.fgeo, cgeo = rand_geo(f, rng), rand_geo(c, rng)
        self.cgeo = GeoData(cgeo.J, cgeo.Jgup_xx, cgeo.Jgup_xy, cgeo.Jgup_yx, cgeo.Jgup_yy, c.dx, c.dy)
        self.cbc = rand_bc(c, [D, N, N, D], [u] * 4, rng)
        self.geo = geo
        if device:
            for k in ("phi", "rhs", "out", "bare", "inv", "xf", "yf", "fine", "crse", "geo", "fgeo", "cgeo"):
                setattr(self, k, getattr(self, k).to_device())

    def arrays(self):
        return [np.asarray(getattr(self, k).host()) for k in
                ("phi", "rhs", "out", "bare", "inv", "xf", "yf", "fine", "crse")]


def _interior(phi):
    """phi's valid cells as an array of their own that shares its memory (leading dimension phi's)."""
    class Inner:
        valid, ngx, ngy, offi, offj = phi.valid, 0, 0, BD_CELL, BD_CELL

        @staticmethod
        def c():
            a = phi.c()
            return type(a)(a.data + 8 * (1 + a.ld), a.ld, 0, 0)
    return Inner


def _same(a):
    """The array behind one descriptor, so that passing it twice passes one pointer twice."""
    class Same:
        valid, ngx, ngy, offi, offj = a.valid, a.ngx, a.ngy, a.offi, a.offj
        one = a.c()

        @staticmethod
        def c():
            return Same.one
    return Same


def _laplacian_onto_itself(M, w):
    p = _same(w.phi)
    M.compute_laplacian(p, p, w.geo, w.bc, False)


def _residual_onto_itself(M, w):
    p = _same(w.phi)
    M.compute_residual(p, w.rhs, p, w.geo, w.bc, False)


CALLS = {
    "laplacian_onto_itself": _laplacian_onto_itself,
    "residual_onto_itself": _residual_onto_itself,
    "residual": lambda M, w: M.compute_residual(w.out, w.rhs, w.phi, w.geo, w.bc, False),
    "residual_into_rhs": lambda M, w: M.compute_residual(w.rhs, w.rhs, w.phi, w.geo, w.bc, False),
    "residual_over_phi": lambda M, w: M.compute_residual(_interior(w.phi), w.rhs, w.phi, w.geo, w.bc, False),
    "residual_of_phi": lambda M, w: M.compute_residual(w.out, _interior(w.phi), w.phi, w.geo, w.bc, False),
    "residual_bare": lambda M, w: M.compute_residual(w.out, w.rhs, w.bare, w.geo, w.bc, True),
    "laplacian": lambda M, w: M.compute_laplacian(w.out, w.phi, w.geo, w.bc, False, True),
    "laplacian_over_phi": lambda M, w: M.compute_laplacian(_interior(w.phi), w.phi, w.geo, w.bc, False),
    "invdiags": lambda M, w: M.compute_invdiags(w.out, w.geo, w.bc, True),
    "fill": lambda M, w: M.fill_ghosts(w.phi, w.bc, w.geo, False),
    "extrapolate": lambda M, w: M.extrapolate_ghosts(w.phi, 2),
    "pd": lambda M, w: M.compute_pd(w.xf, w.phi, 2, 1),
    "grad": lambda M, w: M.compute_grad(w.xf, w.yf, w.phi, w.geo, w.bc, False),
    "boundary_fluxes": lambda M, w: M.fill_boundary_fluxes(w.xf, w.yf, w.bc, False),
    "div": lambda M, w: M.compute_div(w.out, w.xf, w.yf),
    "jacobi": lambda M, w: M.relax_jacobi(w.phi, w.rhs, w.geo, w.bc, False, w.inv, 0.7, -1.0, 3),
    "jacobi_tol": lambda M, w: M.relax_jacobi(w.phi, w.rhs, w.geo, w.bc, False, w.inv, 0.7, 1e-30, 2, True),
    "bicgstab": lambda M, w: M.solve_bicgstab2(w.phi, w.rhs, w.geo, w.bc, True, w.inv, 1e-3, 2, 1, False),
    "restrict": lambda M, w: M.restrict(w.fine, w.crse),
    "prolong1": lambda M, w: M.prolong(w.fine, w.crse, w.fgeo, w.cgeo, w.cbc, 1),
    "prolong2": lambda M, w: M.prolong(w.fine, w.crse, w.fgeo, w.cgeo, w.cbc, 2),
}
for _n in (1, 2, 3, 4, 5):
    CALLS[f"gs{_n}"] = lambda M, w, n=_n: M.relax_gs(w.phi, w.rhs, w.geo, w.bc, False, w.inv, 0.9, -1.0, n, False)
CALLS["gs_rhs_is_phi"] = lambda M, w: M.relax_gs(w.phi, _interior(w.phi), w.geo, w.bc, True, w.inv, 1.0, -1.0, 2, False)
CALLS["gs_tol"] = lambda M, w: M.relax_gs(w.phi, w.rhs, w.geo, w.bc, True, w.inv, 1.0, 1e-30, 3, True)


@pytest.mark.parametrize("call", list(CALLS))
def test_device_arrays_in_place_give_the_bits_of_staged_ones(M, call):
    host, dev = World(False), World(True)
    CALLS[call](M, host)
    CALLS[call](M, dev)
    for a, b in zip(host.arrays(), dev.arrays()):
        assert same(np.ascontiguousarray(a), np.ascontiguousarray(b))


def test_norms_of_device_arrays(M):
    host, dev = World(False), World(True)
    for p in (0, 1, 2):
        assert M.pnorm(host.phi, p) == M.pnorm(dev.phi, p)
    assert M.inner_prod(host.rhs, host.phi) == M.inner_prod(dev.rhs, dev.phi)
    assert M.inner_prod(host.rhs, host.rhs) == M.inner_prod(dev.rhs, dev.rhs)
