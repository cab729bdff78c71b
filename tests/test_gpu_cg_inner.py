"""The complex-symmetric conjugate gradient inner solve of the mixed stage
solver with the element preconditioner: edges of its line passes (one node
pair per line up to the largest degree, even and odd N), partial passes and
blocks, one element, the sign and size of alpha, natural boundaries, and
right-hand sides on which the unconjugated inner product vanishes, where the
preconditioned MINRES has to take over.

The judge is the reference's own test on the true FP64 residual,
|b - A x| < tol |b| + tol (include/minres.hpp:92), with A the oracle's
operator; the two FP64 operators agree to 1e-12, which adds at most
1e-12 |A x| to the left side."""
import numpy as np
import pytest

from tests.util import structured

pytestmark = pytest.mark.gpu
TOL = 1e-10


def _setup(semlib, oracle, n, p, jitter=0.1, neumann=False, resident=True):
    from schrodingersem_gb300 import capi
    co, el = structured(n, box=(-2.0, 2.0, -2.0, 2.0), jitter=jitter, seed=n + p)
    ctx = semlib.Context(p, coords=co, elements=el, neumann=neumann)
    om = oracle.Mesh(p, coords=co, elements=el, neumann=neumann)
    ctx.set_option(capi.OPT_SOLVE_PRECISION, capi.PREC_MIXED)
    ctx.set_option(capi.OPT_PRECOND, capi.PRECOND_FDM)
    ctx.set_option(capi.OPT_RESIDENT, 1 if resident else 0)
    X, Y = om.node_coords()
    return ctx, om, X * X + 2 * Y * Y


def _check(ctx, om, V, alpha, b, maxit=20000):
    xr, xi = ctx.zeros(), ctx.zeros()
    ok, it, _ = ctx.minres_schro(ctx.to_device(V), alpha, xr, xi, ctx.to_device(b[0]), ctx.to_device(b[1]), maxit,
                                 TOL, x_is_zero=True)
    Ax = om.schro_res(V, alpha, xr.cpu().numpy(), xi.cpu().numpy())
    norm = lambda a: np.sqrt(om.dot(a[0], a[0]) + om.dot(a[1], a[1]))  # noqa: E731
    r = norm([b[k] - Ax[k] for k in (0, 1)])
    assert ok and it >= 1
    assert r < TOL * norm(b) + TOL + 1e-12 * norm(Ax), (r, it)
    return it


def _rhs(om, seed):
    rng = np.random.default_rng(seed)
    return [om.mask(om.gproj(rng.standard_normal(om.shape))) for _ in range(2)]


@pytest.mark.parametrize("n,p,resident", [
    (3, 1, False), (5, 2, False), (2, 3, False), (7, 5, False), (1, 8, False), (4, 15, False), (3, 16, False),
    (60, 7, False), (130, 2, False), (1, 8, True), (13, 8, True), (50, 4, True), (33, 6, True), (21, 10, True)])
def test_degrees_and_ragged_passes(semlib, oracle, n, p, resident):
    ctx, om, V = _setup(semlib, oracle, n, p, resident=resident)
    _check(ctx, om, V, 0.004, _rhs(om, 3 * n + p))
    assert (ctx.stats().resident_launches > 0) == resident


@pytest.mark.parametrize("resident", [False, True])
@pytest.mark.parametrize("alpha", [0.0, -0.004, 1e-6, 0.3])
def test_alpha_range(semlib, oracle, alpha, resident):
    ctx, om, V = _setup(semlib, oracle, 12, 6, resident=resident)
    _check(ctx, om, V, alpha, _rhs(om, 5))


@pytest.mark.parametrize("resident", [False, True])
def test_natural_boundary(semlib, oracle, resident):
    ctx, om, V = _setup(semlib, oracle, 9, 8, neumann=True, resident=resident)
    _check(ctx, om, V, 0.004, _rhs(om, 6))


@pytest.mark.parametrize("resident", [False, True])
def test_vanishing_inner_product(semlib, oracle, resident):
    """b = (delta in one element, the same delta in a congruent element far
    away): r.z and p.Ap cancel to rounding in the first iteration"""
    ctx, om, _ = _setup(semlib, oracle, 16, 6, jitter=0.0, resident=resident)
    b = [np.zeros(om.shape), np.zeros(om.shape)]
    b[0][3 * 16 + 4, 3, 2] = 1.0
    b[1][11 * 16 + 9, 3, 2] = 1.0
    _check(ctx, om, np.zeros(om.shape), 0.004, b)


@pytest.mark.parametrize("resident", [False, True])
def test_nan_rhs_is_not_a_solution(semlib, oracle, resident):
    ctx, om, V = _setup(semlib, oracle, 6, 4, resident=resident)
    b = _rhs(om, 7)
    b[0][5, 2, 2] = np.nan
    xr, xi = ctx.zeros(), ctx.zeros()
    ok, _, _ = ctx.minres_schro(ctx.to_device(V), 0.01, xr, xi, ctx.to_device(b[0]), ctx.to_device(b[1]), 50, TOL,
                                x_is_zero=True)
    assert not ok
