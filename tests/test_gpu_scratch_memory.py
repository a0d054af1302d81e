"""Device memory that a context takes for its atoms: the FP64 spread's basis (80 bytes an
atom) only where the tiled spread is taken, the mixed gradient's cotangents (16) only
in the mixed form.  524,288 atoms' worth (capacities are powers of two); allocations
come in pieces of 2 MB, three arrays at most."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, CAP = 300000, 524288
SLACK = 3 * (2 << 20)


def used(call):
    import torch
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    call()
    torch.cuda.synchronize()
    return free - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("M,tiled", [(8, False), (20, True)])
def test_only_what_is_used(M, tiled, precision):
    import torch
    from gse_b200.gse import Context
    fp64 = precision == "fp64"
    rec = 32 if fp64 else 16
    L = 1.0 * M
    ctx = Context(M, M, M, 2.0, 0.4, 3.0, 3.0, L, L, L, precision=precision)
    rng = np.random.default_rng(1)
    x = rng.uniform(0.0, L, (N, 4))
    x[:, 3] = 0.0
    x = torch.from_numpy(x).to(torch.float64 if fp64 else torch.float32).cuda()
    f = torch.zeros(3, N, dtype=torch.float64, device="cuda")
    g = torch.zeros(4, N, dtype=torch.float64, device="cuda")
    ctx.spread_charge(1, x)
    ctx.solve_poisson()
    assert bool(ctx.paths() & 1) == tiled
    want = CAP * (2 * rec + 24 + 12 + (80 if fp64 and tiled else 0))
    got = used(lambda: ctx.spread_charge(N, x))
    assert abs(got - want) <= SLACK, (got, want)
    want = CAP * (56 if fp64 else 72)
    got = used(lambda: ctx.adjoint(N, x, 1.0, None, None, None, g[0], g[1], g[2], g[3]))
    assert abs(got - want) <= SLACK, (got, want)
    # another width's tiled spread finds its basis as well
    if fp64 and not tiled:
        return
    small = x[:500].contiguous()
    small[:, 3] = 1.0
    rho = torch.zeros(M ** 3, dtype=x.dtype, device="cuda")
    ctx.gauss_spread(1.0, 4.0, 500, small, L, L, L, 0, rho)
    assert abs(float(rho.double().sum()) - 500.0) < 1.0
