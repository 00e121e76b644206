"""The work this library is used for, as measurable cases.

A case is a dict of plain values.  ``listed()`` names twelve of them,
``draw(rng)`` gives more of the same ranges; ``prepare(case, seed)`` makes what
a calling program holds before the call (inputs from the seed, geometry,
resident hierarchies), ``run(state)`` makes one pass through the public entry
points, ``work(case)`` counts the bytes and operations a pass cannot do
without, and ``exact(case, seed)`` computes the same outputs in plain torch
FP64 where they have a closed definition: the operator-level calls, and the
solutions of Dirichlet problems small enough for a dense factorisation.

Kinds of case

* ``solve``   -- one solve on a resident hierarchy (api.Solver), device arrays:
  ``solver`` is vcycle (the stationary V-cycle), gmres (GMRES(V-cycle) with the
  exact bottom), fmg or dc (deferred correction); ``mixed`` runs the V-cycle's
  grid levels in FP32.
* ``oneshot`` -- the Fortran-signature vcycle with host arrays: the hierarchy is
  built and freed inside the call, as a program that links the library in
  place of the CPU one makes it.
* ``batch``   -- many independent problems in lockstep (api.Batch).
* ``serve``   -- a burst of requests of different sizes through api.Server with
  resident hierarchies.
* ``op``      -- one operator-level call on device arrays: residual, relax_gs
  (the smoother), project (compute_grad then compute_div).

Maps: identity; wavy (x = xi + 0.1 sin 2 pi xi sin 2 pi eta, y stretched
exponentially to a 64:1 first cell, Dirichlet x and Neumann y sides); skew (y
stretched by a ratio per cell in a wall layer, then sheared; Dirichlet).
"""
import math

import torch

import mgpoisson2d_b200.api as M
from mgpoisson2d_b200.types import (BCMODE_NONUNIFORM, BCTYPE_DIRI, BCTYPE_NEUM, BD_CELL, BD_NODE, BdryData, Box,
                                    BoxData, GeoData)

F64 = torch.float64
DENSE_MOST = 18000   # unknowns solved by a dense factorisation in exact()


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the reference's own problem: 128^2, Cartesian, Dirichlet, plain FP64 V-cycles; a small solve, all latency
        {"name": "vcycle_128", "kind": "solve", "solver": "vcycle", "map": "identity", "nx": 128, "ny": 128,
         "mixed": False},
        # a drop-in call from a CPU program: host arrays, hierarchy built in the call
        {"name": "oneshot_320x192", "kind": "oneshot", "map": "skew", "nx": 320, "ny": 192, "angle": 20.0,
         "ratio": 1.03},
        # the production solver on the stretched grid of the benchmark
        {"name": "gmres_mixed_1024", "kind": "solve", "solver": "gmres", "map": "wavy", "nx": 1024, "ny": 1024,
         "mixed": True},
        # the same solver wholly in FP64, a middle size
        {"name": "gmres_fp64_640x512", "kind": "solve", "solver": "gmres", "map": "wavy", "nx": 640, "ny": 512,
         "mixed": False},
        # sides whose schedule stops early at an odd number (a large bottom level), as requests of any size bring
        {"name": "gmres_mixed_840x432", "kind": "solve", "solver": "gmres", "map": "skew", "nx": 840, "ny": 432,
         "angle": 15.0, "ratio": 1.04, "mixed": True},
        # deferred correction on a large skewed, stretched grid with Dirichlet data
        {"name": "dc_mixed_2048", "kind": "solve", "solver": "dc", "map": "skew", "nx": 2048, "ny": 2048,
         "angle": 30.0, "ratio": 1.05, "mixed": True},
        # deferred correction in FP64, a middle size
        {"name": "dc_fp64_576x352", "kind": "solve", "solver": "dc", "map": "skew", "nx": 576, "ny": 352,
         "angle": 20.0, "ratio": 1.03, "mixed": False},
        # full multigrid from nothing
        {"name": "fmg_512", "kind": "solve", "solver": "fmg", "map": "skew", "nx": 512, "ny": 512, "angle": 10.0,
         "ratio": 1.02, "mixed": False},
        # many uneven problems at once
        {"name": "batch_mixed_32", "kind": "batch", "count": 32, "first": 0, "nmax": 1024, "mixed": True},
        # a burst of requests on a server with resident hierarchies
        {"name": "serve_8", "kind": "serve", "count": 8, "first": 100, "nmax": 512, "mixed": True},
        # the outer residual of a large field
        {"name": "residual_2048", "kind": "op", "op": "residual", "map": "wavy", "nx": 2048, "ny": 2048},
        # a few smoothing sweeps of a small ragged field: the smallest calls a program makes
        {"name": "relax_gs_131x97", "kind": "op", "op": "relax_gs", "map": "skew", "nx": 131, "ny": 97,
         "angle": 12.0, "ratio": 1.02, "sweeps": 4},
    ]


def _log(rng, lo, hi, to=1):
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(max(lo, min(hi, to * round(n / to))))


def draw(rng):
    kind = rng.choice(["op", "op", "solve", "solve", "solve", "oneshot", "batch", "serve"])
    skew = {"angle": round(rng.uniform(0.0, 25.0), 2), "ratio": round(rng.uniform(1.0, 1.05), 4)}
    if kind == "op":
        op = rng.choice(["residual", "relax_gs", "project"])
        c = {"kind": kind, "op": op, "map": rng.choice(["identity", "wavy", "skew"]), "nx": _log(rng, 33, 2048),
             "ny": _log(rng, 33, 2048)}
        if op == "relax_gs":
            c["sweeps"] = rng.choice([1, 2, 4, 8])
        return dict(c, **skew) if c["map"] == "skew" else c
    if kind == "solve":
        solver = rng.choice(["vcycle", "gmres", "gmres", "fmg", "dc"])
        mixed = rng.random() < 0.5 and solver != "fmg"
        if solver == "gmres":
            m = rng.choice(["wavy", "skew"])
            # sides in eighths: even sides down to an odd bottom; on the wavy map whole powers deep
            c = {"kind": kind, "solver": solver, "map": m, "nx": _log(rng, 64, 768, 32 if m == "wavy" else 8),
                 "ny": _log(rng, 64, 768, 32 if m == "wavy" else 8), "mixed": mixed}
        else:
            c = {"kind": kind, "solver": solver, "map": "identity" if rng.random() < 0.3 else "skew",
                 "nx": _log(rng, 64, 1024, 16), "ny": _log(rng, 64, 1024, 16), "mixed": mixed}
        return dict(c, **skew) if c["map"] == "skew" else c
    if kind == "oneshot":
        return {"kind": kind, "map": "skew", "nx": _log(rng, 64, 768, 16), "ny": _log(rng, 64, 768, 16), **skew}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(8, 32), "first": rng.randint(0, 400),
                "nmax": _log(rng, 256, 1024), "mixed": rng.random() < 0.5}
    return {"kind": kind, "count": rng.randint(4, 8), "first": rng.randint(100, 400), "nmax": _log(rng, 128, 512),
            "mixed": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# Geometry and inputs in plain torch
# ---------------------------------------------------------------------------
def _map(case):
    """(xi, eta) -> (x, y) of a case's map."""
    kind = case["map"]
    if kind == "identity":
        return lambda xi, eta: (xi + 0 * eta, eta + 0 * xi)
    if kind == "wavy":
        lo, hi = 1e-9, 60.0
        for _ in range(200):   # beta of a 64:1 first cell
            mid = 0.5 * (lo + hi)
            lo, hi = (mid, hi) if math.expm1(mid) / mid < 64.0 else (lo, mid)
        beta = 0.5 * (lo + hi)

        def wavy(xi, eta):
            x = xi + 0.1 * torch.sin(2 * math.pi * xi) * torch.sin(2 * math.pi * eta)
            return x, torch.expm1(beta * eta) / math.expm1(beta) + 0 * xi
        return wavy
    n, lr, shear = case["ny"], math.log(max(case["ratio"], 1.0 + 1e-9)), math.tan(math.radians(case["angle"]))
    layer = float(min(64, n // 4))

    def prim(t):   # cell heights grow by `ratio` per cell inside the wall layer, linear below 0
        inner = torch.expm1(lr * t.clamp(0.0, layer)) / lr
        return torch.where(t < 0, t, inner + math.exp(lr * layer) * (t - layer).clamp(min=0.0))
    total = float(prim(torch.tensor(float(n), dtype=F64)))

    def skew(xi, eta):
        y = prim(eta * n) / total
        return xi + shear * y, y + 0 * xi
    return skew


def _axis(n, node, ng):
    off = 0.0 if node else 0.5
    return (torch.arange(-ng, n + node + ng, dtype=F64, device="cuda") + off) / n


def _metric(case, node_x, node_y):
    """x_xi, x_eta, y_xi, y_eta of the map by one-cell differences, one ghost layer."""
    nx, ny, f = case["nx"], case["ny"], _map(case)
    xi, eta = _axis(nx, node_x, 1)[None, :], _axis(ny, node_y, 1)[:, None]
    xe, ye = f(xi + 0.5 / nx, eta)
    xw, yw = f(xi - 0.5 / nx, eta)
    xn, yn = f(xi, eta + 0.5 / ny)
    xs, ys = f(xi, eta - 0.5 / ny)
    return (xe - xw) * nx, (xn - xs) * ny, (ye - yw) * nx, (yn - ys) * ny


def _geometry(case):
    """J, J g^ij on cells, x-faces and y-faces as (rows, columns) tensors with one ghost layer."""
    a, b, c, d = _metric(case, 0, 0)
    J = a * d - b * c
    a, b, c, d = _metric(case, 1, 0)
    Jf = a * d - b * c
    xx, xy = (b * b + d * d) / Jf, -(a * b + c * d) / Jf
    a, b, c, d = _metric(case, 0, 1)
    Jf = a * d - b * c
    yx, yy = -(a * b + c * d) / Jf, (a * a + c * c) / Jf
    return [t.contiguous() for t in (J, xx, xy, yx, yy)]


def _types(case):
    return [BCTYPE_DIRI, BCTYPE_DIRI] + [BCTYPE_NEUM if case["map"] == "wavy" else BCTYPE_DIRI] * 2


def _boundary(case, seed):
    """Per side, Dirichlet values (a smooth function of the side) or None: deferred correction takes data."""
    if case.get("solver") != "dc":
        return None
    g = torch.Generator().manual_seed(seed + 77)
    p = torch.rand(4, 2, generator=g, dtype=F64)
    sides = []
    for s in range(4):
        n = case["ny"] if s < 2 else case["nx"]
        t = (torch.arange(n, dtype=F64) + 0.5) / n
        sides.append(torch.cos(2 * math.pi * (t + p[s, 0])) * (0.5 + p[s, 1]))
    return sides


def _rhs(case, J, seed):
    """J (f - <f>_J), f a sum of 16 Fourier modes of the seed at the mapped centres."""
    g = torch.Generator().manual_seed(seed)
    amp = torch.rand(16, generator=g, dtype=F64) * 2 - 1
    mx, my = (torch.randint(1, 9, (16,), generator=g) for _ in range(2))
    x, y = _map(case)(_axis(case["nx"], 0, 0)[None, :], _axis(case["ny"], 0, 0)[:, None])
    f = torch.zeros_like(x)
    for k in range(16):
        f += float(amp[k]) * torch.cos(math.pi * float(mx[k]) * x) * torch.cos(math.pi * float(my[k]) * y)
    Ji = J[1:-1, 1:-1]
    f -= (f * Ji).sum() / Ji.sum()
    return (f if case.get("solver") == "dc" else f * Ji).contiguous()   # dc_vcycle scales by J itself


def _field(case, seed):
    """A smooth field with some noise, ghost ring included: what an operator call meets inside an iteration."""
    g = torch.Generator(device="cuda").manual_seed(seed + 5)
    xi, eta = _axis(case["nx"], 0, 1)[None, :], _axis(case["ny"], 0, 1)[:, None]
    u = torch.sin(2 * math.pi * xi) * torch.cos(3 * math.pi * eta) + 0.3 * torch.cos(5 * xi + 4 * eta)
    return (u + 0.1 * torch.randn(u.shape, generator=g, dtype=F64, device="cuda")).contiguous()


def _pool(case):
    """The problems of a batch or a server: sides log-uniform, a random stretch and shear each."""
    out = []
    for k in range(case["count"]):
        g = torch.Generator().manual_seed(4_000_000 + case["first"] + k)
        u = torch.rand(4, generator=g, dtype=F64).tolist()
        lo, to = (64, 16) if case["kind"] == "batch" else (32, 8)
        side = [math.exp(math.log(lo) + v * (math.log(case["nmax"]) - math.log(lo))) for v in u[:2]]
        nx, ny = (int(max(lo, to * round(n / to))) for n in side)
        out.append({"map": "skew", "nx": nx, "ny": ny, "ratio": 1.0 + 0.06 * u[2], "angle": 25.0 * u[3]})
    return out


# ---------------------------------------------------------------------------
# The library's containers
# ---------------------------------------------------------------------------
def _host(t):
    return t.cpu().numpy().T


def _containers(case, seed, host=False):
    v = Box.of_size(case["nx"], case["ny"])
    J, xx, xy, yx, yy = geo = _geometry(case)
    put = _host if host else (lambda t: t)
    rhs = BoxData(v, data=put(_rhs(case, J, seed)))
    at = [(BD_CELL, BD_CELL), (BD_NODE, BD_CELL), (BD_NODE, BD_CELL), (BD_CELL, BD_NODE), (BD_CELL, BD_NODE)]
    G = GeoData(*[BoxData(v, 1, 1, oi, oj, data=put(t)) for t, (oi, oj) in zip(geo, at)], v.dx, v.dy)
    sides = _boundary(case, seed)
    if sides is None:
        bc = BdryData.uniform(v, _types(case))
    else:
        bc = BdryData(v, _types(case), [BCMODE_NONUNIFORM] * 4, [t.numpy() for t in sides])
    phi = BoxData(v, 1, 1) if host else BoxData.device_zeros(v, 1, 1)
    return {"v": v, "geo": G, "bc": bc, "rhs": rhs, "phi": phi}


def _flags(solver, mixed):
    f = M.FLAG_DIRICHLET_COUPLED_DIAG | (M.FLAG_MIXED if mixed else 0)
    if solver == "gmres":
        f |= M.FLAG_GMRES | M.FLAG_DIRECT_COARSE | M.FLAG_DIRECT_LARGE
    return f


def _inverse_diagonal(case, geo):
    _, xx, _, _, yy = geo
    nx, ny = case["nx"], case["ny"]
    xx, yy = xx[1:-1, 1:-1], yy[1:-1, 1:-1]
    return (-1.0 / ((xx[:, 1:] + xx[:, :-1]) * (nx * nx) + (yy[1:] + yy[:-1]) * (ny * ny))).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        s = _containers(case, seed)
        dd = case["solver"] == "dc"
        s["solver"] = M.Solver(s["v"], s["geo"], s["bc"], M.KIND_DD if dd else M.KIND_MG,
                               _flags(case["solver"], case["mixed"]))
        s["call"] = {"vcycle": s["solver"].vcycle, "gmres": s["solver"].vcycle, "fmg": s["solver"].fmg,
                     "dc": s["solver"].dc_vcycle}[case["solver"]]
    elif kind == "oneshot":
        s = _containers(case, seed, host=True)
    elif kind == "batch":
        s = {"problems": [_containers(dict(p, kind=kind), seed + k) for k, p in enumerate(_pool(case))]}
        s["batch"] = M.Batch([(p["v"], p["geo"], p["bc"]) for p in s["problems"]],
                             flags=_flags("vcycle", case["mixed"]) | M.FLAG_LOCKSTEP, nstreams=8)
    elif kind == "serve":
        s = {"problems": [_containers(dict(p, kind=kind), seed + k) for k, p in enumerate(_pool(case))]}
        s["server"] = M.Server(4, 16 << 30, _flags("gmres", case["mixed"]))
        # a long-running server has its hierarchies resident: one request of each problem, as served before
        tickets = [_submit(s["server"], k, p) for k, p in enumerate(s["problems"])]
        for t in tickets:
            s["server"].wait(t)
    else:
        v = Box.of_size(case["nx"], case["ny"])
        s = _containers(case, seed)
        s["start"] = _field(case, seed)
        s["phi"] = BoxData(v, 1, 1, data=s["start"].clone())
        if case["op"] == "residual":
            s["res"] = BoxData.device_zeros(v)
        elif case["op"] == "relax_gs":
            s["invd"] = BoxData(v, data=_inverse_diagonal(case, _geometry(case)))
        else:
            s["xflux"] = BoxData.device_zeros(v, 0, 0, BD_NODE, BD_CELL)
            s["yflux"] = BoxData.device_zeros(v, 0, 0, BD_CELL, BD_NODE)
            s["div"] = BoxData.device_zeros(v)
    s["case"] = case
    return s


def _submit(server, k, p):
    return server.submit(p["v"], p["geo"], p["bc"], p["phi"], p["rhs"], True, 1e-10, 200, key=k + 1, zerophi=True)


def _inside(phi):
    """The valid cells: the corner ghosts hold a marker, not a result."""
    return phi.data[1:-1, 1:-1]


def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "solve":
        homog = case["solver"] != "dc"
        n = 8
        s["call"](s["phi"], s["rhs"], s["bc"], homog, 1e-10, 300, smooth_down=n, smooth_up=n, smooth_bottom=n,
                  zerophi=True)
        return {"phi": _inside(s["phi"])}
    if kind == "oneshot":
        before = M.set_flags(_flags("vcycle", False))
        M.vcycle(s["phi"], s["rhs"], s["geo"], s["bc"], True, 1e-10, 300, zerophi=True)
        M.set_flags(before)
        return {"phi": _inside(s["phi"])}
    if kind == "batch":
        ps = s["problems"]
        s["batch"].vcycle([p["phi"] for p in ps], [p["rhs"] for p in ps], [p["bc"] for p in ps], True, 1e-10, 300,
                          zerophi=True)
        return {"phi": [_inside(p["phi"]) for p in ps]}
    if kind == "serve":
        tickets = [_submit(s["server"], k, p) for k, p in enumerate(s["problems"])]
        for t in tickets:
            s["server"].wait(t)
        return {"phi": [_inside(p["phi"]) for p in s["problems"]]}
    if case["op"] == "residual":
        M.compute_residual(s["res"], s["rhs"], s["phi"], s["geo"], s["bc"], True)
        return {"res": s["res"].data}
    if case["op"] == "relax_gs":
        s["phi"].data.copy_(s["start"])
        M.relax_gs(s["phi"], s["rhs"], s["geo"], s["bc"], True, s["invd"], 1.0, -1.0, case["sweeps"], False)
        return {"phi": _inside(s["phi"])}
    M.compute_grad(s["xflux"], s["yflux"], s["phi"], s["geo"], s["bc"], True)
    M.compute_div(s["div"], s["xflux"], s["yflux"])
    return {"xflux": s["xflux"].data, "yflux": s["yflux"].data, "div": s["div"].data}


def work(case):
    """Each input read once (rhs, the metric, an iterate where one is given), each output written once, in FP64; the
    operations of one pass of the 9-point operator over the outputs for every sweep or solve asked for."""
    ps = _pool(case) if case["kind"] in ("batch", "serve") else [case]
    cells = float(sum(p["nx"] * p["ny"] for p in ps))
    if case["kind"] != "op":
        return {"bytes": 8 * cells * 7, "flops": 45 * cells}   # rhs, J and the four face arrays in, phi out
    words = {"residual": 7, "relax_gs": 8, "project": 8}[case["op"]]
    return {"bytes": 8 * cells * words, "flops": 45 * cells * case.get("sweeps", 1)}


# ---------------------------------------------------------------------------
# The same outputs in plain torch
# ---------------------------------------------------------------------------
class _Operator:
    """The mapped 9-point operator on a padded field G (valid cells and one ghost ring): the normal differences read the
    ghosts, the transverse ones the quadratic extrapolation of the valid cells."""

    def __init__(self, case, sides=None):
        self.case, self.nx, self.ny = case, case["nx"], case["ny"]
        self.J, self.xx, self.xy, self.yx, self.yy = [t[1:-1, 1:-1] for t in _geometry(case)]
        self.types = _types(case)
        self.sides = [t.cuda() for t in sides] if sides is not None else [0.0] * 4

    def fill(self, G):
        """Third-order Dirichlet ghosts; Neumann ghosts stay as they are."""
        def ghost(g, a, b, c):
            return 3.2 * g - 3.0 * a + b - 0.2 * c
        for s, (at, a, b, c) in enumerate([(0, 1, 2, 3), (-1, -2, -3, -4)] * 2):
            if self.types[s] != BCTYPE_DIRI:
                continue
            if s < 2:
                G[1:-1, at] = ghost(self.sides[s], G[1:-1, a], G[1:-1, b], G[1:-1, c])
            else:
                G[at, 1:-1] = ghost(self.sides[s], G[a, 1:-1], G[b, 1:-1], G[c, 1:-1])
        return G

    def extended(self, G):
        E = G.clone()
        E[1:-1, 0] = 3 * (G[1:-1, 1] - G[1:-1, 2]) + G[1:-1, 3]
        E[1:-1, -1] = 3 * (G[1:-1, -2] - G[1:-1, -3]) + G[1:-1, -4]
        E[0, 1:-1] = 3 * (G[1, 1:-1] - G[2, 1:-1]) + G[3, 1:-1]
        E[-1, 1:-1] = 3 * (G[-2, 1:-1] - G[-3, 1:-1]) + G[-4, 1:-1]
        for j, j1, j2, j3 in ((0, 1, 2, 3), (-1, -2, -3, -4)):
            for i, i1, i2, i3 in ((0, 1, 2, 3), (-1, -2, -3, -4)):
                E[j, i] = 0.5 * (3 * (E[j, i1] - E[j, i2]) + G[j, i3] + 3 * (E[j1, i] - E[j2, i]) + G[j3, i])
        return E

    def fluxes(self, G):
        nx, ny, E = float(self.nx), float(self.ny), self.extended(G)
        ty = E[2:, :] - E[:-2, :]
        tx = E[:, 2:] - E[:, :-2]
        fx = self.xx * (G[1:-1, 1:] - G[1:-1, :-1]) * nx + self.xy * 0.25 * (ty[:, 1:] + ty[:, :-1]) * ny
        fy = self.yy * (G[1:, 1:-1] - G[:-1, 1:-1]) * ny + self.yx * 0.25 * (tx[1:, :] + tx[:-1, :]) * nx
        for s, t in enumerate(self.types):
            if t == BCTYPE_NEUM:   # homogeneous
                (fx if s < 2 else fy.T)[:, 0 if s % 2 == 0 else -1] = 0.0
        return fx, fy

    def div(self, fx, fy):
        return (fx[:, 1:] - fx[:, :-1]) * float(self.nx) + (fy[1:] - fy[:-1]) * float(self.ny)

    def apply(self, G):
        return self.div(*self.fluxes(G))

    def pad(self, phi):
        G = torch.zeros(self.ny + 2, self.nx + 2, dtype=F64, device="cuda")
        G[1:-1, 1:-1] = phi
        return G


def _relax(op, G, rhs, invd, sweeps):
    """Gauss-Seidel sweeps in the library's order: ghosts once, four colours inside, four along the edges, corners."""
    ny, nx = op.ny, op.nx
    i, j = torch.arange(nx, device="cuda")[None, :], torch.arange(ny, device="cuda")[:, None]
    ex, ey = (i == 0) | (i == nx - 1), (j == 0) | (j == ny - 1)
    colours = [(i % 2 == a) & (j % 2 == b) for a, b in ((0, 0), (1, 1), (1, 0), (0, 1))]
    passes = [c & ~ex & ~ey for c in colours] + [c & (ex ^ ey) for c in colours] + [ex & ey]
    for _ in range(sweeps):
        op.fill(G)
        for mask in passes:
            inner = G[1:-1, 1:-1]
            G[1:-1, 1:-1] = torch.where(mask, inner + (rhs - op.apply(G)) * invd, inner)
    return G[1:-1, 1:-1]


def _dense_solution(case, seed):
    """The solution of L[phi] = rhs on a Dirichlet grid: the matrix column by column (impulses far enough apart share a
    probe), then a dense factorisation and one step of refinement."""
    nx, ny = case["nx"], case["ny"]
    n = nx * ny
    op = _Operator(case, _boundary(case, seed))
    rhs = _rhs(case, torch.nn.functional.pad(op.J, (1, 1, 1, 1)), seed)
    if case.get("solver") == "dc":
        rhs = rhs * op.J
    lin = _Operator(case)
    A = torch.zeros(n, n, dtype=F64, device="cuda")
    cells = torch.arange(n, device="cuda").reshape(ny, nx)
    for a in range(7):
        for b in range(7):
            u = torch.zeros(ny, nx, dtype=F64, device="cuda")
            u[b::7, a::7] = 1.0
            out = lin.apply(lin.fill(lin.pad(u)))
            for dj in range(-3, 4):
                for di in range(-3, 4):
                    src = cells[b::7, a::7]
                    jj, ii = src // nx + dj, src % nx + di
                    ok = (jj >= 0) & (jj < ny) & (ii >= 0) & (ii < nx)
                    A[(jj * nx + ii)[ok], src[ok]] = out[jj[ok], ii[ok]]
    lu = torch.linalg.lu_factor(A)

    def solve(r):
        return torch.linalg.lu_solve(*lu, r.reshape(n, 1)).reshape(ny, nx)

    def residual(phi):
        return rhs - op.apply(op.fill(op.pad(phi)))
    phi = solve(residual(torch.zeros(ny, nx, dtype=F64, device="cuda")))
    return phi + solve(residual(phi))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        ps = _pool(case)
        got = [_dense_solution(dict(p, kind=kind), seed + k) if p["nx"] * p["ny"] <= DENSE_MOST // 2 else None
               for k, p in enumerate(ps)]
        return {"phi": got} if any(g is not None for g in got) else None
    if kind in ("solve", "oneshot"):
        if case["map"] == "wavy" or case["nx"] * case["ny"] > DENSE_MOST:
            return None
        return {"phi": _dense_solution(case, seed)}
    op = _Operator(case)
    G = _field(case, seed)
    rhs = _rhs(case, torch.nn.functional.pad(op.J, (1, 1, 1, 1)), seed)
    if case["op"] == "relax_gs":
        return {"phi": _relax(op, G, rhs, _inverse_diagonal(case, _geometry(case)), case["sweeps"])}
    op.fill(G)
    if case["op"] == "residual":
        return {"res": rhs - op.apply(G)}
    fx, fy = op.fluxes(G)
    return {"xflux": fx, "yflux": fy, "div": op.div(fx, fy)}
