"""A tolerance that no residual can meet (zero or negative) runs the conjugate
gradients to max_iter, as the reference's test |r| < tol |b| does
(include/pcg.hpp:84): the same iterates and no success, with the vectors in
shared memory (8 x 8) and streamed (121 x 121)."""
import numpy as np
import pytest

from tests.util import structured

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p", [(8, 4), (121, 6)])
def test_pcg_with_unreachable_tolerance(semlib, n, p):
    co, el = structured(n, box=(-1.0, 1.0, -1.0, 1.0), jitter=0.1, seed=n)
    ctx = semlib.Context(p, coords=co, elements=el)
    X, Y = ctx.node_coords()
    b = ctx.mask(ctx.gproj(ctx.to_device(np.cos(X + Y))))
    out = []
    for tol in (0.0, -1e-6, -1.0):
        x = ctx.zeros()
        ok, it, res = ctx.pcg_laplace(x, b, 25, tol, x_is_zero=True)
        assert not ok and it == 25, tol
        out.append((x.cpu().numpy(), res))
    assert all(np.array_equal(x, out[0][0]) and res == out[0][1] for x, res in out)
