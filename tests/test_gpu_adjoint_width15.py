"""The gradient at stencil width 15, whose kernels run one block per SM, single systems
and a batch against the FP64 form of the same gradient: 2e-5 of the largest component
as in the mixed gradient's other tests (FP32 grids and transforms)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_width15_equals_fp64():
    from gse_b200.gse import Batch, Context
    sizes = [(24, 24, 24), (32, 24, 40), (48, 48, 48)]
    rng = np.random.default_rng(15)
    systems, xs, gs, want = [], [], [], []
    for k, M in enumerate(sizes):
        box = tuple(0.82 * m for m in M)
        n = 300 + 331 * k
        x = np.empty((n, 4))
        x[:, :3] = rng.uniform(-0.1, 1.1, (n, 3)) * np.array(box)
        x[:, 3] = rng.uniform(0.5, 1.0, n) * np.where(np.arange(n) % 2, 1.0, -1.0)
        x = x.astype(np.float32).astype(np.float64)
        g = rng.standard_normal((3, n))
        outs = {}
        for precision in ("fp64", "mixed"):
            ctx = Context(*M, 2.0, 0.4, 3.0, 3.0, *box, precision=precision)
            assert ctx.paths() & 1
            o = np.zeros((4, n))
            ctx.adjoint(n, np.ascontiguousarray(x, dtype=ctx.dtype), 0.7, g[0], g[1], g[2],
                        o[0], o[1], o[2], o[3])
            outs[precision] = o
        w = outs["fp64"]
        scale = np.array([np.abs(w[0]).max()] + [np.abs(w[1:]).max()] * 3)[:, None]
        assert np.all(np.abs(outs["mixed"] - w) <= 2e-5 * scale)
        systems.append({"size": M, "box": box, "n": n})
        xs.append(x), gs.append(g), want.append((w, scale))
    b = Batch(systems, sigma=2.0, kappa=0.4, lambdaSigma1=3.0)
    for fused in (False, True):
        if fused and not b.info().fused_available:
            continue
        b.set_schedule(fused)
        dq, dx = b.adjoint(np.concatenate(xs).astype(np.float32), np.full(3, 0.7),
                           np.concatenate(gs, axis=1).T)
        got = np.concatenate([dq[None], dx.T])
        at = 0
        for w, scale in want:
            assert np.all(np.abs(got[:, at:at + w.shape[1]] - w) <= 2e-5 * scale)
            at += w.shape[1]
