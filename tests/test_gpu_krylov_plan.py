"""Poisson solves on meshes whose share per block comes within the FP64 kernels'
own static arrays (4.2 KB) of the shared memory a block may have: the streamed
form has to take them into account, and the form with its vectors in shared
memory (the last five).  The solve is judged as the library's other conjugate
gradient solves are, by the true residual, 10 tol |b|; an apply follows it, as
an error left behind by the solve would show there."""
import numpy as np
import pytest

from tests.util import rel_err, structured

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p", [(121, 6), (105, 7), (84, 9), (65, 12), (60, 13), (56, 14),
                                 (157, 4), (65, 11), (60, 12), (51, 14), (45, 16)])
def test_poisson_near_the_shared_memory_limit(semlib, oracle, n, p):
    co, el = structured(n, box=(-1.0, 2.0, -0.5, 1.5), jitter=0.2, seed=p + n)
    ctx, om = semlib.Context(p, coords=co, elements=el), oracle.Mesh(p, coords=co, elements=el)
    X, Y = om.node_coords()
    b = om.mask(om.gproj(np.cos(X + Y)))
    x, tol = ctx.zeros(), 1e-6
    ok, _, _ = ctx.pcg_laplace(x, ctx.to_device(b), 20000, tol, x_is_zero=True)
    u = np.random.default_rng(n).standard_normal(om.shape)
    assert rel_err(ctx.apply_laplace(ctx.to_device(u)).cpu().numpy(), om.apply_laplace(u)) <= 1e-12
    r = b - om.apply_laplace(x.cpu().numpy())
    assert ok and np.sqrt(om.dot(r, r)) <= 10 * tol * np.sqrt(om.dot(b, b))
