"""Refinement sweeps of the element-preconditioned stage solve that reduce the true
residual by little, though nothing is wrong with the conjugate gradients: an outer
tolerance below the rounding of the FP64 residual (the sweeps go on to
SEM_OPT_MAX_REFINE), and an inner tolerance near one (many sweeps).  Neither is
handed to MINRES."""
import numpy as np
import pytest

from tests.util import structured

pytestmark = pytest.mark.gpu


def _solve(semlib, resident, tol, **options):
    from schrodingersem_gb300 import capi
    co, el = structured(12, box=(-2.0, 2.0, -2.0, 2.0), jitter=0.1, seed=4)
    ctx = semlib.Context(6, coords=co, elements=el)
    for opt, v in dict(SOLVE_PRECISION=capi.PREC_MIXED, PRECOND=capi.PRECOND_FDM, RESIDENT=resident,
                       **options).items():
        ctx.set_option(getattr(capi, "OPT_" + opt), v)
    rng = np.random.default_rng(5)
    b = [ctx.mask(ctx.unmask(ctx.to_device(rng.standard_normal(ctx.shape)))) for _ in range(2)]
    x = [ctx.zeros(), ctx.zeros()]
    ok, _, res = ctx.minres_schro(ctx.zeros(), 0.004, x[0], x[1], b[0], b[1], 100000, tol, x_is_zero=True)
    return ok, res / np.sqrt(sum(ctx.dot(v, v) for v in b)), ctx.stats()


@pytest.mark.parametrize("resident", [1, 0])
def test_outer_tolerance_below_rounding(semlib, resident):
    ok, rel, st = _solve(semlib, resident, 1e-30, MAX_REFINE=20)
    assert not ok and st.solver_launches == 1 and st.fp64_applies == 21
    assert rel < 1e-12  # the two FP64 operators of a residual agree to 1e-12


@pytest.mark.parametrize("resident", [1, 0])
@pytest.mark.parametrize("inner", [0.5, 0.9])
def test_loose_inner_tolerance(semlib, resident, inner):
    # sweeps reduce by `inner` or better: 1e-8 after at most log(1e-8) / log(inner) = 27, 175 of them
    ok, _, st = _solve(semlib, resident, 1e-8, MAX_REFINE=400, INNER_TOL=inner, ADAPTIVE_INNER=0)
    assert ok and st.solver_launches == 1 and st.fp64_applies <= 2 + np.log(1e-8) / np.log(inner)
