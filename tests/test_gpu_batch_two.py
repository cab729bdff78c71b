"""Ensembles created side by side: the second one's kernels (same degree, less
shared memory) are prepared before the first one's step is captured, and must
not take the first one's shared memory from it.  Both give the bits that each
gives alone."""
import numpy as np
import pytest

from tests.util import structured

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", [2, 0])
def test_ensembles_side_by_side(semlib, precond):
    from schrodingersem_gb300 import capi
    from schrodingersem_gb300.batch import Batch
    from schrodingersem_gb300.meshgen import gaussian_packet

    def instance(n, p):
        h = 0.2 * n + 1.0
        co, el = structured(n, box=(-h, h, -h, h), jitter=0.1, seed=n)
        ctx = semlib.Context(p, coords=co, elements=el)
        X, Y = ctx.node_coords()
        re, im = gaussian_packet(X, Y, (0.1, -0.2), 0.4 * h, (1.5, -1.0))
        return (p, co, el), re, im, np.ascontiguousarray(X * X)

    def step(B, f):
        re, im = f[1].copy(), f[2].copy()
        assert B.bdf2([re], [im], [f[3]], 0.004, 5e-3, 100000, 1e-10) == [True]
        return re, im

    def make(f):
        B = Batch([f[0]])
        B.set_option(capi.OPT_PRECOND, precond)
        return B

    fields = [instance(12, 8), instance(2, 8)]
    alone = [step(make(f), f) for f in fields]
    batches = [make(f) for f in fields]
    for B, f, ref in zip(batches, fields, alone):
        got = step(B, f)
        assert all(np.array_equal(a, b) for a, b in zip(got, ref))
