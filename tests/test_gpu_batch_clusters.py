"""Batched instances on clusters of 1, 2, 4 and 8 blocks (by their node count)
against the single-instance FP64 driver: sizes on both sides of the limits
4,096, 8,192 and 16,384 nodes, odd node counts (the FP32 vectors are read as
pairs), shares that do not divide the elements evenly, with the element
preconditioner (conjugate gradients) and without (MINRES on one block).

Both sides stop on |r| < tol (|r0| + 1); at tol = 1e-10 the library's tests
bound the difference of the states by 1e-8, and the error is proportional to
the residual: 1e-9 at tol = 1e-11."""
import numpy as np
import pytest

from tests.util import rel_err, structured

pytestmark = pytest.mark.gpu

SIZES = [(8, 7), (8, 8), (6, 12), (8, 11), (6, 19), (4, 25), (8, 15), (4, 1), (5, 3), (2, 9)]


@pytest.mark.parametrize("precond", [2, 0])
def test_cluster_sizes_match_single_instance(semlib, precond):
    from schrodingersem_gb300 import capi
    from schrodingersem_gb300.batch import Batch
    from schrodingersem_gb300.meshgen import gaussian_packet
    dt, steps, tol = 5e-3, 2, 1e-11
    T = (steps - 0.5) * dt
    meshes, fields, ref = [], [], []
    for q, (p, n) in enumerate(SIZES if precond else SIZES[:5]):
        h = 0.2 * n + 1.0
        co, el = structured(n, box=(-h, h, -h, h), jitter=0.1, seed=q)
        ctx = semlib.Context(p, coords=co, elements=el)
        X, Y = ctx.node_coords()
        re, im = gaussian_packet(X, Y, (0.1, -0.2), 0.4 * h, (1.5, -1.0))
        V = X * X + 0.5 * Y * Y
        a, b = re.copy(), im.copy()
        assert ctx.schrodinger("bdf2", a, b, V, T, dt, 100000, tol)
        meshes.append((p, co, el))
        fields.append((re.copy(), im.copy(), np.ascontiguousarray(V)))
        ref.append((a, b))
    B = Batch(meshes)
    B.set_option(capi.OPT_PRECOND, precond)
    re, im, V = ([f[k] for f in fields] for k in range(3))
    assert all(B.bdf2(re, im, V, T, dt, 100000, tol))
    for i in range(len(meshes)):
        assert B.instance(i)[0] == steps and B.instance(i)[2] > 0
        assert max(rel_err(re[i], ref[i][0]), rel_err(im[i], ref[i][1])) < 1e-9, (i, SIZES[i])
