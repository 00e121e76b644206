"""Solvers and batches are made, used and freed by one thread while another has a stream
capture under way (a program's own CUDA graph, or another solver's first V-cycle): the
capture and both threads' results stand."""
from __future__ import annotations

import threading

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


def _problem(n=64):
    v = Box.of_size(n, n)
    geo = G.mapped_geometry(v, G.map_skew_stretch(15.0, 1.02, 0.25, n))
    return v, geo, rand_field(v, np.random.default_rng(n), 0), BdryData(v, [D] * 4, [BCMODE_UNIFORM] * 4)


def _free_solver(M, p):
    v, geo, rhs, bc = p
    s = M.Solver(v, geo, bc, KIND_MG, 0)
    s.vcycle(BoxData(v, 1, 1), rhs, bc, True, 1e-6, 3)
    return s.close


def _free_batch(M, p):
    v, geo, rhs, bc = p
    b = M.Batch([(v, geo, bc)] * 2, KIND_MG, M.FLAG_LOCKSTEP | M.FLAG_DIRICHLET_COUPLED_DIAG)
    b.vcycle([BoxData(v, 1, 1) for _ in range(2)], [rhs, rhs], [bc, bc], True, 1e-6, 3)
    return b.close


def _one_shot(M, p):
    v, geo, rhs, bc = p
    return lambda: M.vcycle(BoxData(v, 1, 1), rhs, geo, bc, True, 1e-6, 3)


def _operators(M, p):
    v, geo, rhs, bc = p

    def work():
        res, phi, inv = BoxData(v), BoxData(v, 1, 1), BoxData(v)
        M.compute_invdiags(inv, geo, bc, True)
        M.relax_gs(phi, rhs, geo, bc, True, inv, 1.0, 0.0, 3, True)
        M.compute_residual(res, rhs, phi, geo, bc, True)
        assert 0.0 < M.pnorm(res, 2) < M.pnorm(rhs, 2)
    return work


def _map(M, p):
    return lambda: M.map_geometry(p[0], M.MAP_IDENTITY, device=False)


@pytest.mark.parametrize("make", [_free_solver, _free_batch, _one_shot, _operators, _map])
def test_a_capture_in_another_thread_stands(M, make):
    work = make(M, _problem())
    x = torch.zeros(1000, device="cuda")
    g, st, errors = torch.cuda.CUDAGraph(), torch.cuda.Stream(), []

    def other():
        torch.cuda.set_device(0)
        try:
            work()
        except Exception as e:
            errors.append(e)

    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        x.add_(1.0)
        t = threading.Thread(target=other)
        t.start()
        t.join()
        x.mul_(2.0)
    assert not errors, errors
    x.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.all(x == 2.0)


def test_solvers_of_eight_threads(M):
    problems = [_problem(n) for n in (40, 48, 56, 64, 72, 80, 96, 104)]

    def solve(p):
        v, geo, rhs, bc = p
        out = []
        for flags in (0, M.FLAG_MIXED, M.FLAG_KRYLOV, M.FLAG_GMRES | M.FLAG_DIRECT_COARSE):
            with M.Solver(v, geo, bc, KIND_MG, flags) as s:
                phi = BoxData(v, 1, 1)
                s.vcycle(phi, rhs, bc, True, 1e-8, 6)
            out.append(phi.interior().copy())
            phi = BoxData(v, 1, 1)
            M.vcycle(phi, rhs, geo, bc, True, 1e-8, 2)
            out.append(phi.interior().copy())
        return out

    want = [solve(p) for p in problems]
    errors = []

    def run(k):
        torch.cuda.set_device(0)
        try:
            for _ in range(4):
                for a, b in zip(want[k], solve(problems[k])):
                    assert np.array_equal(a, b)
        except Exception as e:
            errors.append((k, e))

    threads = [threading.Thread(target=run, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
