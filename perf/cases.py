"""Timed workloads of the library: what a program has it do, through the
public Python classes (``Context``, ``Batch``, ``Learner``).

A case is a dict of plain values with a ``kind``:

  apply      one operator apply into buffers the caller owns
  solve      one linear solve from a zero guess (MINRES on the stage operator,
             or the Poisson / Helmholtz drivers), FP64
  steps      a few time steps of a Schroedinger driver from the same state
  batch      a few BDF2 steps of an ensemble of independent small meshes
  forward    inference of the stage-guess network on all elements of a mesh
  gradient   loss and gradients of one minibatch of its training

``prepare`` holds what such a program keeps (mesh context, fields, network),
``run`` is one pass, ``exact`` the same outputs from plain FP64 torch: its own
quadrature, geometry, assembly and solvers on the global nodes.
Meshes are n x n jittered quads in row order; Dirichlet nodes hold zero.
"""
import math

import numpy as np
import torch

import schrodingersem_gb300 as S
from schrodingersem_gb300 import capi
from schrodingersem_gb300.batch import Batch
from schrodingersem_gb300.learned import Learner
from schrodingersem_gb300.meshgen import structured_quads

SIDE = 0.25  # element side of the time-stepping meshes (64 elements on [-8, 8])
DT = 5e-3    # their time step
OPS = ("res", "f", "laplace", "helmholtz", "gproj")


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest call: one FP64 operator apply on a coarse mesh, as a user's own iteration makes it
        {"name": "apply_small", "kind": "apply", "op": "res", "dtype": "f64", "n": 8, "p": 4},
        # FP64 operator apply of a large mesh (stage operator, both components)
        {"name": "apply_f64", "kind": "apply", "op": "res", "dtype": "f64", "n": 256, "p": 8},
        # FP32 operator apply of a larger one, odd element count
        {"name": "apply_f32", "kind": "apply", "op": "res", "dtype": "f32", "n": 301, "p": 8},
        # FP64 MINRES on the stage operator: the default precision of every Schroedinger driver
        {"name": "minres_f64", "kind": "solve", "op": "res", "n": 64, "p": 8},
        # Poisson driver (PCG), mid-size odd mesh
        {"name": "poisson", "kind": "solve", "op": "laplace", "n": 45, "p": 6},
        # Helmholtz driver (MINRES), high degree
        {"name": "helmholtz", "kind": "solve", "op": "helmholtz", "n": 32, "p": 12},
        # a small run with the default options (FP64, zero stage guess): 256 elements of degree 4
        {"name": "steps_small", "kind": "steps", "method": "dirk4s3", "form": "fp64", "n": 16, "p": 4, "steps": 2},
        # the fast form on the 64 x 64 mesh: FP32 inner solve, element preconditioner, projected stage guess
        {"name": "steps_project", "kind": "steps", "method": "dirk4s3", "form": "project", "n": 64, "p": 8, "steps": 4},
        # a mesh too large to stay on chip: five-stage method, extrapolated stage guess
        {"name": "steps_large", "kind": "steps", "method": "dirk4s5", "form": "extrapolate", "n": 192, "p": 8,
         "steps": 2},
        # ensemble of independent instances, n in 4..32 and p in {4, 6, 8}
        {"name": "batch", "kind": "batch", "count": 160, "n_max": 32, "steps": 2},
        # network inference for the 4096 elements of the 64 x 64 mesh at p = 8
        {"name": "forward", "kind": "forward", "rows": 4096, "p": 8, "hidden": 256},
        # one minibatch of its training
        {"name": "gradient", "kind": "gradient", "rows": 1024, "p": 8, "hidden": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "solve", "solve", "steps", "steps", "batch", "forward", "gradient"])
    if kind == "apply":
        dtype = rng.choice(["f64", "f32"])
        op = "res" if dtype == "f32" else rng.choice(OPS)
        p = rng.randint(2, 16)
        top = 301 * 9 if dtype == "f32" else 256 * 9
        return {"kind": kind, "op": op, "dtype": dtype, "n": _log_int(rng, 4, top // (p + 1)), "p": p}
    if kind == "solve":
        op = rng.choice(["res", "laplace", "helmholtz"])
        p = rng.randint(3, 12)
        return {"kind": kind, "op": op, "n": _log_int(rng, 4, (64 if op == "res" else 48) * 9 // (p + 1)), "p": p}
    if kind == "steps":
        form = rng.choice(["fp64", "zero", "extrapolate", "project"])
        p = rng.randint(3, 12)
        top = 24 if form == "fp64" else 128
        return {"kind": kind, "method": rng.choice(["dirk4s3", "dirk4s5", "bdf2"]), "form": form,
                "n": _log_int(rng, 4, top * 9 // (p + 1)), "p": p, "steps": rng.randint(2, 3)}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 8, 160), "n_max": rng.randint(6, 32), "steps": rng.randint(1, 2)}
    p = rng.choice([4, 6, 8])
    return {"kind": kind, "rows": _log_int(rng, 100, 4096 if kind == "forward" else 1024), "p": p,
            "hidden": rng.choice([64, 128, 256])}


# ------------------------------------------------- plain FP64 discretisation
def _lgl(p):
    x = -np.cos(np.pi * np.arange(p + 1) / p)
    P = np.polynomial.legendre
    c = np.zeros(p + 1)
    c[p] = 1.0
    d1, d2 = P.legder(c), P.legder(c, 2)
    for _ in range(50):
        x[1:-1] -= P.legval(x[1:-1], d1) / P.legval(x[1:-1], d2)
    return x, 2.0 / (p * (p + 1) * P.legval(x, c) ** 2)


def _dmatrix(x):
    N = len(x)
    b = np.array([1.0 / np.prod(x[i] - np.delete(x, i)) for i in range(N)])
    D = np.zeros((N, N))
    for i in range(N):
        for j in range(N):
            if i != j:
                D[i, j] = b[j] / b[i] / (x[i] - x[j])
        D[i, i] = -D[i].sum()
    return D


class _Mesh:
    """Element-local operators of n x n quads in row order, on global nodes."""

    def __init__(self, n, p, coords, elements, dev="cuda", full=True):
        self.n, self.p, self.N, N = n, p, p + 1, p + 1
        z, w = _lgl(p)
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
        co = t(coords)[torch.as_tensor(elements.astype(np.int64), device=dev)]  # E, 4, 2
        xi, eta = t(z)[None, None, :], t(z)[None, :, None]
        c = lambda k, d: co[:, k, d][:, None, None]  # noqa: E731
        self.X, self.Y = (0.25 * (c(0, d) * (1 - xi) * (1 - eta) + c(1, d) * (1 + xi) * (1 - eta)
                                  + c(2, d) * (1 + xi) * (1 + eta) + c(3, d) * (1 - xi) * (1 + eta)) for d in (0, 1))
        q = torch.arange(n * n, device=dev)
        j, i = torch.arange(N, device=dev)[:, None], torch.arange(N, device=dev)[None, :]
        self.width = n * p + 1
        self.gid = (((q // n) * p)[:, None, None] + j) * self.width + ((q % n) * p)[:, None, None] + i
        g = torch.arange(self.width ** 2, device=dev)
        r, s = g // self.width, g % self.width
        self.inside = ((r > 0) & (r < self.width - 1) & (s > 0) & (s < self.width - 1)).double()
        if not full:
            return
        # the copy that holds a shared node's value: its first element in row order
        e = q[:, None, None].expand(-1, N, N)
        first = torch.full((self.width ** 2,), n * n, device=dev, dtype=torch.long)
        first.scatter_reduce_(0, self.gid.reshape(-1), e.reshape(-1), "amin")
        self.owner = (first[self.gid] == e).double()
        self.D = t(_dmatrix(z))
        ww = t(w)[None, None, :] * t(w)[None, :, None]
        d_xi = lambda d: 0.25 * ((1 - eta) * (c(1, d) - c(0, d)) + (1 + eta) * (c(2, d) - c(3, d)))  # noqa: E731
        d_eta = lambda d: 0.25 * ((1 - xi) * (c(3, d) - c(0, d)) + (1 + xi) * (c(2, d) - c(1, d)))  # noqa: E731
        xx, yx, xe, ye = d_xi(0), d_xi(1), d_eta(0), d_eta(1)
        J = xx * ye - xe * yx
        # the discretisation's own metric: y_xi enters the third factor at the transposed node
        yt = 0.25 * ((1 - xi) * (c(1, 1) - c(0, 1)) + (1 + xi) * (c(2, 1) - c(3, 1)))
        self.g11 = ww * (ye * ye + xe * xe) / J
        self.g12 = ww * (ye * yx + xe * xx) / J
        self.g22 = ww * (yt * yt + xx * xx) / J
        self.m = ww * J

    def scatter(self, a):
        o = torch.zeros(self.width ** 2, dtype=a.dtype, device=a.device)
        return o.index_add_(0, self.gid.reshape(-1), a.reshape(-1)) * self.inside

    def glob(self, a):  # element-local continuous field -> global nodes
        o = torch.zeros(self.width ** 2, dtype=a.dtype, device=a.device)
        o[self.gid.reshape(-1)] = a.reshape(-1)
        return o

    def masked(self, g):  # global nodes -> element-local, owner copies only
        return g[self.gid] * self.owner

    def stiff(self, g, mass=None):
        """assembled (K + M c) g, c an element-local field"""
        u, D = g[self.gid], self.D.to(g.dtype)
        ur, us = u @ D.T, torch.matmul(D, u)
        o = (self.g11 * ur - self.g12 * us) @ D + torch.matmul(D.T, self.g22 * us - self.g12 * ur)
        return self.scatter(o if mass is None else o + self.m * mass * u)

    def lump(self):
        return self.scatter(self.m) + (1 - self.inside)


def _krylov(A, b, dg, tol=1e-14):
    """conjugate residuals of the (complex) symmetric A, scaled by dg, restarted on the true residual"""
    x, n0 = torch.zeros_like(b), float(torch.linalg.vector_norm(b))
    best = None
    for _ in range(6):
        r = b - A(x)
        rn = float(torch.linalg.vector_norm(r))
        if best is None or rn < 0.5 * best[0]:
            best = (rn, x.clone())
        else:
            break
        if rn <= tol * n0:
            break
        z = r / dg
        p, Az = z.clone(), A(z)
        q, rho = Az.clone(), (z * Az).sum()
        for it in range(1, 4000):
            Pq = q / dg
            a = rho / (q * Pq).sum()
            x = x + a * p
            r = r - a * q
            z = z - a * Pq
            if it % 16 == 0 and float(torch.linalg.vector_norm(r)) < max(1e-12 * rn, 0.3 * tol * n0):
                break
            Az = A(z)
            new = (z * Az).sum()
            p, q, rho = z + (new / rho) * p, Az + (new / rho) * q, new
    return best[1]


def _stage(M, V, alpha, br, bi):
    """[M, aL; aL, -M] (u, v) = (br, bi) as (M + i a L)(u - i v) = br + i bi"""
    lump = M.lump()
    w = _krylov(lambda q: (lump * M.inside) * q + 1j * alpha * M.stiff(q, V), torch.complex(br, bi), lump + 0j)
    return w.real.contiguous(), -w.imag.contiguous()


GAMMA = math.cos(math.pi / 18) / math.sqrt(3) + 0.5
DELTA = 1 / (6 * (2 * GAMMA - 1) ** 2)
TABLEAU = {
    "dirk4s3": (GAMMA, [[], [0.5 - GAMMA], [2 * GAMMA, 1 - 4 * GAMMA]], [DELTA, 1 - 2 * DELTA, DELTA]),
    "dirk4s5": (0.25, [[], [0.5], [17 / 50, -1 / 25], [371 / 1360, -137 / 2720, 15 / 544],
                       [25 / 24, -49 / 48, 125 / 16, -85 / 12]], [25 / 24, -49 / 48, 125 / 16, -85 / 12, 0.25]),
}


def _advance(M, method, u, v, V, steps):
    hist = []
    for k in range(steps):
        if method == "bdf2":
            lump = M.lump()
            hist.append((lump * u, -lump * v))
            if k == 0:
                (br, bi), alpha = hist[0], DT
            else:
                br, bi = (4 / 3 * hist[-1][q] - 1 / 3 * hist[-2][q] for q in (0, 1))
                alpha = 2 / 3 * DT
            u, v = _stage(M, V, alpha, br, bi)
            continue
        g, rows, wts = TABLEAU[method]
        zs = []
        for row in rows:
            a = u + sum(c * z[0] for c, z in zip(row, zs))
            b = v + sum(c * z[1] for c, z in zip(row, zs))
            zs.append(_stage(M, V, g * DT, -DT * M.stiff(b, V), -DT * M.stiff(a, V)))
        u, v = (s + sum(c * z[q] for c, z in zip(wts, zs)) for q, s in ((0, u), (1, v)))
    return u, v


# ------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _box(case):
    h = 0.5 * SIDE * case["n"] if case["kind"] == "steps" or (case["kind"] == "solve" and case["op"] == "res") else 1.0
    return (-h, h, -h, h)


def _coords(case):
    return structured_quads(case["n"], box=_box(case), jitter=0.1, seed=1)


def _packet(M, rnd, half):
    """normalised-size wave packet (zero on the boundary) and a harmonic trap with three bumps; rnd: uniform(0, 1) list"""
    X, Y = M.X, M.Y
    cx, cy = (0.4 * half * (2 * r - 1) for r in rnd[:2])
    s, kx, ky = (0.15 + 0.1 * rnd[2]) * half, 6 * rnd[3] - 3, 6 * rnd[4] - 3
    amp = torch.exp(-((X - cx) ** 2 + (Y - cy) ** 2) / (2 * s * s)) * M.inside[M.gid]
    V = X * X + Y * Y
    for b in range(3):
        a, w, x0, y0 = rnd[5 + 4 * b:9 + 4 * b]
        V = V + 40 * (a - 0.5) * torch.exp(-((X - half * (2 * x0 - 1)) ** 2 + (Y - half * (2 * y0 - 1)) ** 2)
                                           / (2 * (0.1 * half * (1 + w)) ** 2))
    ph = kx * X + ky * Y
    return (amp * torch.cos(ph)).contiguous(), (amp * torch.sin(ph)).contiguous(), V.contiguous()


def _fields(case, M, seed):
    g = _gen(seed)
    kind, op = case["kind"], case.get("op")
    if kind == "steps" or (kind == "solve" and op == "res"):
        re, im, V = _packet(M, torch.rand(17, generator=g, device="cuda", dtype=torch.float64).tolist(), _box(case)[1])
        return {"re": re, "im": im, "V": V}
    if kind == "solve":
        k = (1 + 3 * torch.rand(4, generator=g, device="cuda", dtype=torch.float64)).tolist()
        return {"f": torch.sin(k[0] * M.X + 1) * torch.cos(k[1] * M.Y) * k[2] + k[3],
                "c": 5 * k[2] * (1 + 0.5 * torch.sin(k[3] * M.X) * torch.cos(k[0] * M.Y))}
    dt = torch.float32 if case["dtype"] == "f32" else torch.float64
    out = {}
    for name in ("u", "v"):
        r = torch.randn(M.width ** 2, generator=g, device="cuda", dtype=torch.float64) * M.inside
        out[name] = r[M.gid].to(dt).contiguous()
    out["V"] = (5 * torch.rand(M.X.shape, generator=g, device="cuda", dtype=torch.float64)).to(dt)
    return out


def _instances(case):
    rng = np.random.default_rng(2026)
    out = []
    for _ in range(case["count"]):
        n, p = int(rng.integers(4, case["n_max"] + 1)), int(rng.choice([4, 6, 8]))
        out.append((n, p) + structured_quads(n, box=(-6.0, 6.0, -6.0, 6.0), jitter=0.1, seed=int(rng.integers(1 << 30))))
    return out


def _batch_fields(insts, seed, full):
    rnd = torch.rand(len(insts), 17, generator=_gen(seed), device="cuda", dtype=torch.float64).tolist()
    ms = [_Mesh(n, p, co, el, full=full) for n, p, co, el in insts]
    return ms, [_packet(M, r, 6.0) for M, r in zip(ms, rnd)]


def _net(case, seed):
    N2 = (case["p"] + 1) ** 2
    d_in, H, d_out = 4 * N2, case["hidden"], 2 * N2
    g = _gen(seed)
    x = torch.randn(case["rows"], d_in, generator=g, device="cuda").to(torch.bfloat16)
    t = torch.randn(case["rows"], d_out, generator=g, device="cuda")
    rng = np.random.default_rng(7)  # the trained network a program keeps
    params = [((rng.standard_normal((i, o)) * math.sqrt(2 / i)).astype(np.float32),
               (0.1 * rng.standard_normal(o)).astype(np.float32)) for i, o in ((d_in, H), (H, H), (H, d_out))]
    return x, t, params


# --------------------------------------------------------------- prepare, run
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forward", "gradient"):
        x, t, params = _net(case, seed)
        L = Learner(x.shape[1], case["hidden"], t.shape[1])
        for k, (W, b) in enumerate(params):
            L.set_params(k, W, b)
        return {"case": case, "net": L, "x": x, "t": t}
    if kind == "batch":
        insts = _instances(case)
        _, f = _batch_fields(insts, seed, False)
        B = Batch([(p, co, el) for _, p, co, el in insts])
        return {"case": case, "B": B, "re0": [a[0] for a in f], "im0": [a[1] for a in f], "V": [a[2] for a in f],
                "re": [torch.empty_like(a[0]) for a in f], "im": [torch.empty_like(a[0]) for a in f]}
    co, el = _coords(case)
    ctx = S.Context(case["p"], coords=co, elements=el)
    M = _Mesh(case["n"], case["p"], co, el, full=False)
    st = {"case": case, "ctx": ctx, **_fields(case, M, seed)}
    if kind == "steps":
        if case["form"] != "fp64":
            ctx.set_option(capi.OPT_SOLVE_PRECISION, capi.PREC_MIXED)
            ctx.set_option(capi.OPT_PRECOND, capi.PRECOND_FDM)
            ctx.set_option(capi.OPT_STAGE_GUESS, capi.GUESS_ZERO if case["form"] == "zero" else capi.GUESS_EXTRAPOLATE)
            ctx.set_option(capi.OPT_PROJECT, 16 if case["form"] == "project" else 0)
        st["a"], st["b"] = torch.empty_like(st["re"]), torch.empty_like(st["re"])
    elif kind == "solve":
        if case["op"] == "res":
            br, bi = ctx.schro_f(st["V"], st["re"], st["im"])
            st["br"], st["bi"] = DT * br, DT * bi
            st["xi"] = torch.empty_like(br)
        st["xr"] = torch.empty_like(M.X)
    else:
        st["yr"], st["yi"] = torch.empty_like(st["u"]), torch.empty_like(st["u"])
    return st


TOL = 1e-12       # relative and absolute residual of every solve: its own error stays small beside the outputs
ALPHA_APPLY = 0.01


def run(st):
    case = st["case"]
    kind, op = case["kind"], case.get("op")
    if kind == "forward":
        return st["net"].forward(st["x"])
    if kind == "gradient":
        loss = st["net"].train_step(st["x"], st["t"], lr=0.0)
        return [loss] + [st["net"].grads(k) for k in range(3)]
    if kind == "batch":
        for k in range(len(st["re"])):
            st["re"][k].copy_(st["re0"][k])
            st["im"][k].copy_(st["im0"][k])
        st["B"].bdf2(st["re"], st["im"], st["V"], (case["steps"] - 0.5) * DT, DT, 100000, TOL)
        return [torch.cat([a.reshape(-1) for a in st[k]]) for k in ("re", "im")]
    ctx = st["ctx"]
    if kind == "steps":
        a, b = st["a"].copy_(st["re"]), st["b"].copy_(st["im"])
        ctx.schrodinger(case["method"], a, b, st["V"], (case["steps"] - 0.5) * DT, DT, 100000, TOL)
        return [a, b]
    if kind == "solve":
        x = st["xr"].zero_()
        if op == "res":
            ctx.minres_schro(st["V"], GAMMA * DT, x, st["xi"].zero_(), st["br"], st["bi"], 100000, TOL, x_is_zero=True)
            return [x, st["xi"]]
        if op == "laplace":
            ctx.poisson(x, st["f"], 100000, TOL)
        else:
            ctx.helmholtz(x, st["c"], st["f"], 100000, TOL)
        return [x]
    u, v, V, yr, yi = (st[k] for k in ("u", "v", "V", "yr", "yi"))
    if op == "res":
        return list((ctx.schro_res_f32 if case["dtype"] == "f32" else ctx.schro_res)(V, ALPHA_APPLY, u, v, yr, yi))
    if op == "f":
        return list(ctx.schro_f(V, u, v, yr, yi))
    if op == "laplace":
        return [ctx.apply_laplace(u, yr)]
    if op == "helmholtz":
        return [ctx.apply_helmholtz(V, u, yr)]
    return [ctx.gproj(u, yr)]


# ------------------------------------------------------------------- floors
def work(case):
    """bytes each input and output needs once and the operations of the plain
    line contractions; an iterative solve counts its operator applies and
    vectors at a nominal iteration count of its size"""
    kind, op = case["kind"], case.get("op")
    if kind in ("forward", "gradient"):
        N2, H, R = (case["p"] + 1) ** 2, case["hidden"], case["rows"]
        w = 4 * N2 * H + H * H + 2 * N2 * H
        if kind == "forward":
            return {"bytes": R * (8 * N2 + 8 * N2) + 2 * w, "flops": 2.0 * R * w}
        return {"bytes": R * (8 * N2 + 8 * N2) + 8 * w, "flops": 6.0 * R * w}
    if kind == "batch":
        loc = sum(n * n * (p + 1) ** 2 for n, p, _, _ in _instances(case))
        return {"bytes": loc * case["steps"] * 8.0 * 12, "flops": loc * case["steps"] * 2.0 * (16 * 8 + 23) * 40}
    N = case["p"] + 1
    loc = float(case["n"] ** 2 * N * N)
    two = op in ("res", "f") or kind == "steps"
    apply = loc * ((16 * N + 23) if two else (8 * N + 12) if op != "gproj" else 1)
    if kind == "apply":
        words = {"res": 9, "f": 9, "laplace": 5, "helmholtz": 7, "gproj": 3}[op]
        return {"bytes": loc * words * (4 if case["dtype"] == "f32" else 8), "flops": apply}
    if kind == "solve":
        its = {"res": 40 * N * N, "laplace": 2.5 * case["n"] * N, "helmholtz": 5 * case["n"] * N}[op]
        return {"bytes": loc * 8 * (9 if two else 7), "flops": apply * its}
    stages = {"dirk4s3": 3, "dirk4s5": 5, "bdf2": 1}[case["method"]] * case["steps"]
    its = 40 * N * N if case["form"] == "fp64" else 5 * N
    return {"bytes": loc * 8 * 9 * stages, "flops": apply * its * stages}


# -------------------------------------------------------------------- exact
def exact(case, seed):
    kind, op = case["kind"], case.get("op")
    if kind in ("forward", "gradient"):
        x, t, params = _net(case, seed)
        ps = [tuple(torch.as_tensor(a, dtype=torch.float64, device="cuda") for a in q) for q in params]
        h = [x.double()]
        for k, (W, b) in enumerate(ps):
            o = h[-1] @ W + b
            h.append(torch.relu(o) if k < 2 else o)
        if kind == "forward":
            return h[3]
        d = h[3] - t.double()
        grads, g = [None] * 3, 2 * d / d.numel()
        for k in (2, 1, 0):
            grads[k] = (h[k].T @ g, g.sum(0))
            if k:
                g = (g @ ps[k][0].T) * (h[k] > 0)
        return [float((d * d).mean())] + grads
    if kind == "batch":
        return _exact_batch(case, seed)
    co, el = _coords(case)
    M = _Mesh(case["n"], case["p"], co, el)
    f = _fields(case, M, seed)
    if kind == "apply":
        u, v, V = (f[k].double() for k in ("u", "v", "V"))
        gu, gv = M.glob(u), M.glob(v)
        if op == "gproj":
            return [M.masked(M.lump() * gu * M.inside)]
        if op in ("laplace", "helmholtz"):
            return [M.masked(M.stiff(gu, V if op == "helmholtz" else None))]
        Lu, Lv = M.stiff(gu, V), M.stiff(gv, V)
        if op == "f":
            return [M.masked(-Lv), M.masked(-Lu)]
        lump = M.lump()
        return [M.masked(lump * gu + ALPHA_APPLY * Lv), M.masked(ALPHA_APPLY * Lu - lump * gv)]
    if kind == "solve":
        if op == "res":
            u, v = M.glob(f["re"]), M.glob(f["im"])
            x, y = _stage(M, f["V"], GAMMA * DT, -DT * M.stiff(v, f["V"]), -DT * M.stiff(u, f["V"]))
            return [M.masked(x), M.masked(y)]
        c = f["c"] if op == "helmholtz" else None
        dg = M.scatter(M.m if c is None else M.m * (1 + c)) + (1 - M.inside)
        dg = dg + M.scatter(M.g11 * (M.D ** 2).sum(0)[None, None, :] + M.g22 * (M.D ** 2).sum(0)[None, :, None])
        return [M.masked(_krylov(lambda q: M.stiff(q, c), M.scatter(M.m * f["f"]), dg))]
    if case["n"] * case["p"] > 64 * 8:
        return None  # a plain solve of these takes too long
    u, v = _advance(M, case["method"], M.glob(f["re"]), M.glob(f["im"]), f["V"], case["steps"])
    return [u[M.gid], v[M.gid]]


def _exact_batch(case, seed):
    insts = _instances(case)
    ms, f = _batch_fields(insts, seed, True)
    out = [None] * len(insts)
    for p in (4, 6, 8):  # the instances of one degree as one disconnected mesh
        idx = [k for k, q in enumerate(insts) if q[1] == p]
        if not idx:
            continue
        U = _Mesh.__new__(_Mesh)
        off = np.concatenate([[0], np.cumsum([ms[k].width ** 2 for k in idx])])
        U.gid = torch.cat([ms[k].gid + int(o) for k, o in zip(idx, off)])
        for a in ("g11", "g12", "g22", "m"):
            setattr(U, a, torch.cat([getattr(ms[k], a) for k in idx]))
        U.inside, U.D = torch.cat([ms[k].inside for k in idx]), ms[idx[0]].D
        size = int(off[-1])

        def scatter(a, U=U, size=size):
            o = torch.zeros(size, dtype=a.dtype, device=a.device)
            return o.index_add_(0, U.gid.reshape(-1), a.reshape(-1)) * U.inside
        U.scatter = scatter
        re, im, V = (torch.cat([f[k][q] for k in idx]) for q in range(3))
        u, v = (torch.zeros(size, dtype=torch.float64, device="cuda") for _ in range(2))
        u[U.gid.reshape(-1)], v[U.gid.reshape(-1)] = re.reshape(-1), im.reshape(-1)
        u, v = _advance(U, "bdf2", u, v, V, case["steps"])
        u, v, e = u[U.gid], v[U.gid], 0
        for k in idx:
            ne = insts[k][0] ** 2
            out[k] = (u[e:e + ne].reshape(-1), v[e:e + ne].reshape(-1))
            e += ne
    return [torch.cat([o[q] for o in out]) for q in (0, 1)]
