"""A forward call replayed on page-locked host memory, after that memory has become
pageable at the same address (unregistered here; a freed block given out again looks
the same): the call then copies as it does for any pageable array and gives what a
fresh context gives, bit for bit, and registered again it is replayed again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRAPH = 4  # GSE_PATH_GRAPH


@pytest.mark.parametrize("explicit", [False, True])
@pytest.mark.parametrize("which", ["xyzq", "forces"])
def test_replay_looks_host_memory_up_again(which, explicit):
    import torch
    from gse_b200 import workloads as W
    from gse_b200.gse import Context
    n, L, M = 600, 20.0, 20
    rt = torch.cuda.cudart()

    def context():
        ctx = Context(M, M, M, 2.0, 0.4, 3.0, 3.0, L, L, L, precision="mixed")
        if explicit:
            ctx.stream = torch.cuda.Stream()
            ctx.set_stream(ctx.stream.cuda_stream)
        return ctx

    def register(a):
        assert int(rt.cudaHostRegister(a.ctypes.data, a.nbytes, 0)) == 0

    def unregister(a):
        assert int(rt.cudaHostUnregister(a.ctypes.data)) == 0

    x0 = W.triplets(n, L, 3)
    x, f = x0.copy(), np.zeros((3, n))
    register(x)
    register(f)
    ctx = context()

    def check(shift):
        x[:] = x0
        x[:, 0] += np.float32(shift)
        f[:] = 0.0
        e = ctx.forward(n, x, f[0], f[1], f[2])
        g = np.zeros((3, n))
        assert context().forward(n, x.copy(), g[0], g[1], g[2]) == e
        assert np.array_equal(f, g)

    for k in range(4):
        check(0.125 * k)
    assert ctx.paths() & GRAPH
    moved = x if which == "xyzq" else f
    unregister(moved)
    check(0.75)
    assert not ctx.paths() & GRAPH
    check(1.0)
    register(moved)
    for k in range(8):
        check(0.125 * k)
    assert ctx.paths() & GRAPH
    unregister(x)
    unregister(f)
