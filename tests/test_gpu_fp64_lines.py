"""FP64 kernels on parity-split lines, where their dispatch and tiling turn:
applies on both sides of the size limits (ragged element counts) and their ring
pass, Krylov solves with vectors in shared memory and streamed, from one element
to more elements than fit; the projection's grouped dot products at basis sizes
around the groups of 8; network GEMMs whose leading dimensions allow only narrow
loads."""
import numpy as np
import pytest

from tests.util import rel_err, structured

pytestmark = pytest.mark.gpu


def _pair(semlib, oracle, n, p):
    co, el = structured(n, box=(-1.0, 2.0, -0.5, 1.5), jitter=0.2, seed=p + n)
    return semlib.Context(p, coords=co, elements=el), oracle.Mesh(p, coords=co, elements=el)


# two components: from 1e5 nodes at p >= 8, from 4e5 at p = 6, 7
@pytest.mark.parametrize("n,p", [(35, 8), (36, 8), (32, 9), (25, 12), (24, 12), (19, 16), (18, 16), (91, 6), (80, 7)])
def test_two_component_applies(semlib, oracle, n, p):
    """the library's FP64 operator tolerance, 1e-12 relative"""
    ctx, om = _pair(semlib, oracle, n, p)
    rng = np.random.default_rng(n * p)
    u, v, V = (rng.standard_normal(om.shape) for _ in range(3))
    d = [ctx.to_device(a) for a in (V, u, v)]
    for got, want in ((ctx.schro_res(d[0], 0.0123, d[1], d[2]), om.schro_res(V, 0.0123, u, v)),
                      (ctx.schro_f(*d), om.schro_f(V, u, v))):
        for k in (0, 1):
            assert rel_err(got[k].cpu().numpy(), want[k]) <= 1e-12


# one component: from 1e6 nodes at p >= 6
@pytest.mark.parametrize("n,p", [(111, 8), (112, 8), (143, 6), (77, 12)])
def test_one_component_applies(semlib, oracle, n, p):
    ctx, om = _pair(semlib, oracle, n, p)
    rng = np.random.default_rng(n * p)
    u, c = (rng.standard_normal(om.shape) for _ in range(2))
    du, dc = ctx.to_device(u), ctx.to_device(c)
    assert rel_err(ctx.apply_laplace(du).cpu().numpy(), om.apply_laplace(u)) <= 1e-12
    assert rel_err(ctx.apply_helmholtz(dc, du).cpu().numpy(), om.apply_helmholtz(c, u)) <= 1e-12


# the ring pass gives corners threads of their own up to 311,296 items (3 n^2 + 4 n + 1 at p = 2)
@pytest.mark.parametrize("n,p", [(3, 2), (321, 2), (322, 2), (330, 2), (140, 8)])
def test_ring_pass_same_bits(semlib, n, p):
    """in place of its input an apply is assembled by the gather over all nodes
    instead of the ring pass: the same sums in the same order"""
    co, el = structured(n, jitter=0.2, seed=n)
    ctx = semlib.Context(p, coords=co, elements=el)
    u = ctx.to_device(np.random.default_rng(n).standard_normal(ctx.shape))
    out = ctx.apply_laplace(u)
    ctx.apply_laplace(u, u)
    assert bool((out == u).all())


@pytest.mark.parametrize("n,p", [(1, 4), (40, 1), (13, 8), (5, 15), (13, 16), (64, 8), (100, 8)])
def test_krylov_forms(semlib, oracle, n, p):
    """MINRES stops on its recurrence's |r| < tol |b| + tol, conjugate gradients
    on theirs.  After k iterations of MINRES the true residual is off by at most
    3 sqrt(3) k eps |A| |x| (the leading part of the bound of Sleijpen, van der
    Vorst and Modersitzki, SIAM J. Matrix Anal. Appl. 22, 2000); conjugate
    gradients get the library's factor 10 for their own norm.  The largest stage
    systems need more than maxit iterations: there the true residual has to be
    the reported one"""
    ctx, om = _pair(semlib, oracle, n, p)
    rng = np.random.default_rng(n + p)
    X, Y = om.node_coords()
    smooth = [om.mask(om.gproj(np.cos((k + 1) * X + Y) + 0.1 * rng.standard_normal(om.shape))) for k in (0, 1)]
    norm = lambda *a: np.sqrt(sum(om.dot(q, q) for q in a))  # noqa: E731
    db = [ctx.to_device(b) for b in smooth]
    tol, maxit = 1e-6, 20000
    V = X * X + Y * Y
    x = [ctx.zeros(), ctx.zeros()]
    ok, it, res = ctx.minres_schro(ctx.to_device(V), 0.004, *x, *db, maxit, tol, x_is_zero=True)
    A = om.schro_res(V, 0.004, *(q.cpu().numpy() for q in x))
    limit = tol * norm(*smooth) + tol if ok else res
    assert ok or it == maxit + 1
    assert norm(*(smooth[k] - A[k] for k in (0, 1))) <= 1.01 * limit
    y = ctx.zeros()
    c = np.full(om.shape, -20.0)
    w = om.mask(om.global_sum(rng.standard_normal(om.shape)))
    for _ in range(30):  # |A| by power iterations
        w = om.mask(om.apply_helmholtz(c, w / norm(w)))
    ok, it, _ = ctx.minres_helmholtz(ctx.to_device(c), y, db[0], maxit, tol, x_is_zero=True)
    y = y.cpu().numpy()
    drift = 3 * np.sqrt(3.0) * it * 2.0 ** -53 * norm(w) * norm(y)
    assert ok and norm(smooth[0] - om.apply_helmholtz(c, y)) <= 1.01 * (tol * norm(smooth[0]) + tol) + drift
    y = ctx.zeros()
    ok, _, _ = ctx.pcg_laplace(y, db[0], maxit, tol, x_is_zero=True)
    assert ok and norm(smooth[0] - om.apply_laplace(y.cpu().numpy())) <= 10 * tol * norm(smooth[0])


@pytest.mark.parametrize("K", [1, 7, 8, 9, 24])
def test_projection_basis_sizes(semlib, K):
    """tolerance of the projection's own test: 1e-8 at tol = 1e-10"""
    from schrodingersem_gb300 import capi
    from schrodingersem_gb300.meshgen import gaussian_packet
    co, el = structured(7, box=(-3.0, 3.0, -3.0, 3.0), jitter=0.1, seed=5)
    ctx = semlib.Context(5, coords=co, elements=el)
    X, Y = ctx.node_coords()
    re, im = gaussian_packet(X, Y, (-0.5, 0.0), 0.8, (2.0, 0.5))
    V = X * X + Y * Y
    steps, dt, tol = 10, 0.01, 1e-10
    a = [re.copy(), im.copy()]
    assert ctx.schrodinger("dirk4s3", *a, V, steps * dt, dt, 100000, tol)
    for opt, val in ((capi.OPT_SOLVE_PRECISION, capi.PREC_MIXED), (capi.OPT_PRECOND, capi.PRECOND_FDM),
                     (capi.OPT_REFINE_TOL_SCALE, 0.1), (capi.OPT_STAGE_GUESS, 1), (capi.OPT_PROJECT, K)):
        ctx.set_option(opt, val)
    b = [re.copy(), im.copy()]
    rec = []
    assert ctx.schrodinger("dirk4s3", *b, V, steps * dt, dt, 100000, tol, record=rec)
    assert ctx.stats().projected_guesses == 3 * len(rec) - 1  # every stage but the very first
    assert max(rel_err(b[0], a[0]), rel_err(b[1], a[1])) < 1e-8


@pytest.mark.parametrize("d_in,hidden,d_out", [(37, 33, 19), (34, 46, 22), (36, 44, 52), (200, 136, 72)])
def test_gradients_at_narrow_leading_dimensions(semlib, d_in, hidden, d_out):
    """tolerances of the two GEMM paths' comparison at even widths"""
    from schrodingersem_gb300 import capi
    from schrodingersem_gb300.learned import Learner
    import torch
    L = capi.load()
    g = torch.Generator(device="cuda").manual_seed(d_in)
    X = torch.randn(300, d_in, generator=g, device="cuda").to(torch.bfloat16)
    T = torch.randn(300, d_out, generator=g, device="cuda")
    out = []
    try:
        for path in (0, 1):
            capi.check(L.sem_gemm_set_path(path), "sem_gemm_set_path")
            net = Learner(d_in, hidden, d_out, seed=5)
            out.append((net.train_step(X, T, lr=0.0), [q for l in range(3) for q in net.grads(l)]))
    finally:
        capi.check(L.sem_gemm_set_path(1), "sem_gemm_set_path")
    assert abs(out[0][0] - out[1][0]) <= 1e-5 * abs(out[0][0])
    for a, b in zip(out[0][1], out[1][1]):
        assert np.abs(a - b).max() <= 1e-4 * max(np.abs(a).max(), 1e-12)
