"""Stage solves whose residual stays above its smallest value for hundreds of
iterations (a potential well with alpha |V| = 25, a random potential with
alpha |V| up to 80): the conjugate gradients go on to convergence and do not hand
the solve to MINRES.  Success means the reference's test on the true FP64 residual
(include/minres.hpp:92)."""
import numpy as np
import pytest

from tests.util import structured

pytestmark = pytest.mark.gpu
TOL = 1e-9


@pytest.mark.parametrize("resident", [1, 0])
@pytest.mark.parametrize("case", ["well", "random"])
def test_long_plateau(semlib, oracle, case, resident):
    from schrodingersem_gb300 import capi
    co, el = structured(32, box=(-4.0, 4.0, -4.0, 4.0), jitter=0.1, seed=1)
    ctx, om = semlib.Context(8, coords=co, elements=el), oracle.Mesh(8, coords=co, elements=el)
    for opt, v in ((capi.OPT_SOLVE_PRECISION, capi.PREC_MIXED), (capi.OPT_PRECOND, capi.PRECOND_FDM),
                   (capi.OPT_RESIDENT, resident)):
        ctx.set_option(opt, v)
    X, Y = om.node_coords()
    rng = np.random.default_rng(3)
    V, alpha = (-1e4 * (np.abs(X) < 1.2), 0.0025) if case == "well" else (1e3 * rng.standard_normal(om.shape), 0.02)
    b = [om.mask(om.gproj(np.exp(-9 * (X * X + Y * Y) / 16) * f)) for f in (np.cos(9 * X / 4), np.sin(9 * X / 4))]
    xr, xi = ctx.zeros(), ctx.zeros()
    ok, _, _ = ctx.minres_schro(ctx.to_device(V), alpha, xr, xi, ctx.to_device(b[0]), ctx.to_device(b[1]), 20000, TOL,
                                x_is_zero=True)
    st = ctx.stats()
    assert ok and st.solver_launches == 1 and st.resident_launches == resident
    Ax = om.schro_res(V, alpha, xr.cpu().numpy(), xi.cpu().numpy())
    norm = lambda a: np.sqrt(om.dot(a[0], a[0]) + om.dot(a[1], a[1]))  # noqa: E731
    assert norm([b[k] - Ax[k] for k in (0, 1)]) < TOL * norm(b) + TOL + 1e-12 * norm(Ax)
