"""The per-atom arrays at the capacities where they go from one allocation to six and back
(powers of two from 1024 on), in contexts that grow to them: energy, forces and gradient
from host arrays, which all the arrays take part in, are the same bits as in a context
that had room for twice as many from its first call (the mixed form's sums are integer,
the FP64 form's run in a fixed order; its gradient's source is left out)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def call(ctx, x, gradient):
    n = len(x)
    f, d = np.zeros((3, n)), np.zeros((4, n))
    e = ctx.forward(n, x, f[0], f[1], f[2])
    if gradient:
        g = np.sin(np.arange(3.0 * n)).reshape(3, n)
        ctx.adjoint(n, x, 0.5, g[0], g[1], g[2], d[0], d[1], d[2], d[3])
    return np.concatenate([[e], f.ravel(), d.ravel()])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_growing_contexts(precision):
    from gse_b200.gse import Context
    box = (20.0, 21.0, 23.0)

    def context():
        return Context(20, 21, 23, 2.0, 0.4, 3.0, 3.0, *box, precision=precision)

    def charges(n):
        rng = np.random.default_rng(n)
        x = np.empty((n, 4), dtype=np.float64 if precision == "fp64" else np.float32)
        x[:, :3] = rng.uniform(0.0, 1.0, (n, 3)) * np.array(box)
        x[:, 3] = rng.uniform(0.5, 1.0, n) * np.where(np.arange(n) % 2, 1.0, -1.0)
        return x

    roomy, grown = context(), context()
    call(roomy, charges(70000), False)
    for n in (1024, 1025, 8192, 8193, 16384, 16385, 32768, 32769, 65536):
        x = charges(n)
        want = call(roomy, x, precision == "mixed")
        assert np.array_equal(call(grown, x, precision == "mixed"), want)
        assert np.array_equal(call(context(), x, precision == "mixed"), want)
