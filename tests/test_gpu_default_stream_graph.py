"""Repeated calls on the legacy default stream replay a graph, in order with the work
around them on that stream, and a program that changes its buffers is left alone.
Replays run the kernels of the direct call, so results are equal bit for bit."""
import pytest

pytestmark = pytest.mark.gpu

GRAPH = 4  # GSE_PATH_GRAPH


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_default_stream_replays_in_order(precision):
    import torch
    from gse_b200 import workloads as W
    from gse_b200.gse import Context
    n, L, M = 600, 20.0, 20
    dt = torch.float64 if precision == "fp64" else torch.float32
    x0 = torch.from_numpy(W.triplets(n, L, 3)).to(dt).cuda()

    def context():
        return Context(M, M, M, 2.0, 0.4, 3.0, 3.0, L, L, L, precision=precision)

    def evaluate(ctx, x):
        f = torch.zeros(3, n, dtype=torch.float64, device="cuda")
        e = torch.zeros(1, dtype=torch.float64, device="cuda")
        ctx.forward(n, x, f[0], f[1], f[2], energy_out=e)
        return torch.cat([e, f.reshape(-1)])

    ctx, x = context(), x0.clone()
    f = torch.zeros(3, n, dtype=torch.float64, device="cuda")
    e = torch.zeros(1, dtype=torch.float64, device="cuda")
    got = []
    for k in range(6):  # no wait between the update, the call and the copies
        x.copy_(x0)
        x[:, 0] += 0.125 * k
        ctx.forward(n, x, f[0], f[1], f[2], energy_out=e)
        got.append(torch.cat([e, f.reshape(-1)]))
    assert ctx.paths() & GRAPH
    for k in range(6):
        x = x0.clone()
        x[:, 0] += 0.125 * k
        want = evaluate(context(), x)
        assert torch.equal(got[k], want), k
    # the same stream again keeps the graph, another drops it
    ctx.set_stream(0)
    assert ctx.paths() & GRAPH
    side = torch.cuda.Stream()
    ctx.set_stream(side.cuda_stream)
    assert not ctx.paths() & GRAPH
    # buffers that change every few calls: right results, however often it captures
    ctx = context()
    bufs = [x0.clone(), x0 + 0.25]
    want = [evaluate(context(), b.to(dt)) for b in bufs]
    outs = [(torch.zeros_like(f), torch.zeros_like(e)) for _ in bufs]
    for k in range(40):
        b = k // 4 % 2
        ctx.forward(n, bufs[b], outs[b][0][0], outs[b][0][1], outs[b][0][2], energy_out=outs[b][1])
        assert torch.equal(torch.cat([outs[b][1], outs[b][0].reshape(-1)]), want[b])
