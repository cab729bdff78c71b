"""The preconditioned MINRES that takes over when the conjugate gradients of the
element-preconditioned stage solve give up: from the on-chip kernel, from the
streaming one and inside an ensemble's cluster (1, 4 and 8 blocks).

The takeover is forced through the inner tolerance: at 1e-30 its square is zero in
FP32, so the conjugate gradients cannot reach it and end by breakdown or stall.
The solve is judged as every mixed solve is, by the true FP64 residual; the
refinement sweeps of both iterations together stay within SEM_OPT_MAX_REFINE.

The ensemble's inner tolerance follows the outer one, so there the outer one is
out of reach as well (success is False) and the states are compared with the
single-instance FP64 driver at tol = 1e-11, bound 1e-9 as in
test_gpu_batch_clusters.py: sweeps that reduce by all that FP32 holds (1e-6 or
better) leave less than tol |r0| after two."""
import numpy as np
import pytest

from tests.util import rel_err, structured

pytestmark = pytest.mark.gpu
TOL = 1e-10


def _forced(semlib, n, p, resident, cap):
    from schrodingersem_gb300 import capi
    co, el = structured(n, box=(-2.0, 2.0, -2.0, 2.0), jitter=0.1, seed=n + p)
    ctx = semlib.Context(p, coords=co, elements=el)
    for opt, v in ((capi.OPT_SOLVE_PRECISION, capi.PREC_MIXED), (capi.OPT_PRECOND, capi.PRECOND_FDM),
                   (capi.OPT_RESIDENT, resident), (capi.OPT_INNER_TOL, 1e-30), (capi.OPT_ADAPTIVE_INNER, 0),
                   (capi.OPT_MAX_REFINE, cap)):
        ctx.set_option(opt, v)
    return ctx, co, el


@pytest.mark.parametrize("n,p,resident", [(12, 6, 1), (12, 6, 0), (9, 5, 0), (5, 8, 1), (70, 8, 0)])
def test_minres_takes_over_and_solves(semlib, oracle, n, p, resident):
    ctx, co, el = _forced(semlib, n, p, resident, 50)
    om = oracle.Mesh(p, coords=co, elements=el)
    rng = np.random.default_rng(n * p)
    b = [om.mask(om.gproj(rng.standard_normal(om.shape))) for _ in range(2)]
    V = rng.uniform(0.0, 4.0, om.shape)
    xr, xi = ctx.zeros(), ctx.zeros()
    ok, _, _ = ctx.minres_schro(ctx.to_device(V), 0.004, xr, xi, ctx.to_device(b[0]), ctx.to_device(b[1]), 100000, TOL,
                                x_is_zero=True)
    st = ctx.stats()
    assert ok and st.solver_launches == 2 and st.resident_launches == resident
    Ax = om.schro_res(V, 0.004, xr.cpu().numpy(), xi.cpu().numpy())
    norm = lambda a: np.sqrt(om.dot(a[0], a[0]) + om.dot(a[1], a[1]))  # noqa: E731
    assert norm([b[k] - Ax[k] for k in (0, 1)]) < TOL * norm(b) + TOL + 1e-12 * norm(Ax)


@pytest.mark.parametrize("resident", [1, 0])
@pytest.mark.parametrize("cap", [1, 3])
def test_sweeps_of_both_iterations_stay_within_the_cap(semlib, resident, cap):
    ctx, _, _ = _forced(semlib, 12, 6, resident, cap)
    rng = np.random.default_rng(3)
    b = [ctx.mask(ctx.unmask(ctx.to_device(rng.standard_normal(ctx.shape)))) for _ in range(2)]
    x = [ctx.zeros(), ctx.zeros()]
    ok, _, _ = ctx.minres_schro(ctx.zeros(), 0.004, x[0], x[1], b[0], b[1], 100000, 1e-30, x_is_zero=True)
    st = ctx.stats()
    # one FP64 apply per sweep and one final residual per launch
    assert not ok and st.solver_launches == 2 and st.fp64_applies - st.solver_launches <= cap


@pytest.mark.parametrize("cap", [2, 6])
def test_takeover_in_a_cluster(semlib, cap):
    from schrodingersem_gb300 import capi
    from schrodingersem_gb300.batch import Batch
    from schrodingersem_gb300.meshgen import gaussian_packet
    dt = 5e-3
    meshes, fields, ref = [], [], []
    for q, (p, n) in enumerate([(8, 15), (8, 11), (5, 3)]):
        h = 0.2 * n + 1.0
        co, el = structured(n, box=(-h, h, -h, h), jitter=0.1, seed=q)
        ctx = semlib.Context(p, coords=co, elements=el)
        X, Y = ctx.node_coords()
        re, im = gaussian_packet(X, Y, (0.1, -0.2), 0.4 * h, (1.5, -1.0))
        V = np.ascontiguousarray(X * X + 0.5 * Y * Y)
        a, b = re.copy(), im.copy()
        assert ctx.schrodinger("bdf2", a, b, V, 0.5 * dt, dt, 100000, 1e-11)
        meshes.append((p, co, el))
        fields.append((re, im, V))
        ref.append((a, b))

    def run(inner_tol, tol, refine):
        B = Batch(meshes)
        B.set_option(capi.OPT_INNER_TOL, inner_tol)
        B.set_option(capi.OPT_MAX_REFINE, refine)
        re, im = [f[0].copy() for f in fields], [f[1].copy() for f in fields]
        ok = B.bdf2(re, im, [f[2] for f in fields], 0.5 * dt, dt, 100000, tol)
        return ok, re, im, [B.instance(i)[2] for i in range(len(meshes))]

    ok, _, _, cg = run(1e-4, 1e-11, 50)
    assert all(ok)
    ok, re, im, its = run(1e-30, 1e-30, cap)
    for i in range(len(meshes)):
        assert not ok[i] and its[i] > 3 * cg[i], (i, its[i], cg[i])  # MINRES needs several times CG's iterations
        if cap > 2:
            assert max(rel_err(re[i], ref[i][0]), rel_err(im[i], ref[i][1])) < 1e-9, i
