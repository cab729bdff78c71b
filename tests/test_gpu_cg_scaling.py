"""The element-preconditioned stage solve does not depend on the unit of length:
with coordinates scaled by 2^k, alpha by 4^k and V by 4^-k the stage operator is
4^k times the unscaled one in exact arithmetic and, powers of two being exact,
in floating point too, so the same right-hand side takes the same iterations to
the same digits.  k reaches the elements whose squared FP32 measure is still a
normal number (2^-126 < m^2 < 2^127, the preconditioner's own range): the inner
products of the recurrence then lie between 1e-21 and 1e+20, and their squares
outside FP32's range."""
import numpy as np
import pytest

from tests.util import structured

pytestmark = pytest.mark.gpu


def _solve(semlib, n, p, k, resident):
    from schrodingersem_gb300 import capi
    co, el = structured(n, box=(-1.0, 1.0, -1.0, 1.0), jitter=0.1, seed=n)
    s = 2.0 ** k
    ctx = semlib.Context(p, coords=co * s, elements=el)
    ctx.set_option(capi.OPT_SOLVE_PRECISION, capi.PREC_MIXED)
    ctx.set_option(capi.OPT_PRECOND, capi.PRECOND_FDM)
    ctx.set_option(capi.OPT_RESIDENT, resident)
    rng = np.random.default_rng(n + p)
    V = rng.uniform(0.0, 2.0, ctx.shape) / (s * s)
    b = [ctx.mask(ctx.unmask(ctx.to_device(rng.standard_normal(ctx.shape)))) for _ in range(2)]
    x = [ctx.zeros(), ctx.zeros()]
    ok, it, res = ctx.minres_schro(ctx.to_device(V), 0.004 * s * s, x[0], x[1], b[0], b[1], 20000, 1e-9, x_is_zero=True)
    return ok, it, res, ctx.stats().solver_launches, [t.cpu().numpy() * (s * s) for t in x]


@pytest.mark.parametrize("resident", [0, 1])
@pytest.mark.parametrize("k", [-28, -20, 12, 25, 28])
def test_unit_of_length(semlib, k, resident):
    ok, it, res, launches, x = _solve(semlib, 6, 6, 0, resident)
    assert ok and launches == 1
    sk = _solve(semlib, 6, 6, k, resident)
    assert sk[:4] == (ok, it, res, launches)
    assert np.array_equal(sk[4][0], x[0]) and np.array_equal(sk[4][1], x[1])
