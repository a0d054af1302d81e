"""A replayed forward call among calls that share its grids, bins and Green's table: the
table follows the box of each call, and gradient, virial and the separate calls leave
what the next replay needs.  Every result has to be that of a fresh context which makes
the one call alone, bit for bit: a replay runs the kernels of the direct call, and their
sums run in fixed orders (the mixed form's are integer sums).  Only the FP64 gradient's
source is summed by atomics, some 165 terms a grid point at most: 1e-11 of its largest
component holds 165 roundings at cancellations of a thousand; a wrong box moves it by a
hundredth."""
import pytest

pytestmark = pytest.mark.gpu

GRAPH = 4  # GSE_PATH_GRAPH
OWN_FFT = 8  # GSE_PATH_OWN_FFT
N = 600
# (form, grid side): cuFFT with and without the callback plan, and the own FFT
GRIDS = [("fp64", 20), ("fp64", 64), ("mixed", 20), ("mixed", 64)]


class Run:
    def __init__(self, precision, M, box):
        import torch
        from gse_b200 import workloads as W
        from gse_b200.gse import Context
        self.ctx = Context(M, M, M, 2.0, 0.4, 3.0, 3.0, *box, precision=precision)
        dt = torch.float64 if precision == "fp64" else torch.float32
        self.x = torch.from_numpy(W.triplets(N, 20.0, 3)).to(dt).cuda()
        self.x[:, :3] *= M / 20.0
        self.f = torch.zeros(3, N, dtype=torch.float64, device="cuda")
        self.e = torch.zeros(1, dtype=torch.float64, device="cuda")

    def forward(self):
        import torch
        self.ctx.forward(N, self.x, self.f[0], self.f[1], self.f[2], energy_out=self.e)
        return torch.cat([self.e, self.f.reshape(-1)])

    def adjoint(self):
        import torch
        g = torch.linspace(-1, 1, 3 * N, dtype=torch.float64, device="cuda").reshape(3, N)
        out = torch.zeros(4, N, dtype=torch.float64, device="cuda")
        self.ctx.adjoint(N, self.x, 0.5, g[0], g[1], g[2], out[0], out[1], out[2], out[3])
        return out.reshape(-1)

    def virial(self):
        import torch
        self.ctx.spread_charge(N, self.x)
        out = torch.zeros(6, dtype=torch.float64, device="cuda")
        self.ctx.virial(out)
        return out

    def separate(self):
        import torch
        self.ctx.spread_charge(N, self.x)
        self.ctx.solve_poisson()
        f = torch.zeros(3, N, dtype=torch.float64, device="cuda")
        self.ctx.interpolate_force(N, self.x, f[0], f[1], f[2])
        return f.reshape(-1)

    def virial_after_forward(self):
        import torch
        out = torch.zeros(6, dtype=torch.float64, device="cuda")
        self.ctx.virial(out)
        return out


def same(got, want, atomics):
    import torch
    if atomics:
        return bool((got - want).abs().max() <= 1e-11 * want.abs().max())
    return torch.equal(got, want)


@pytest.mark.parametrize("between", ["adjoint", "virial", "separate"])
@pytest.mark.parametrize("precision,M", GRIDS)
def test_replay_after_a_call_in_another_box(precision, M, between):
    import torch
    A, B = (1.0 * M,) * 3, (1.02 * M, 0.99 * M, 1.01 * M)
    want = Run(precision, M, A).forward()
    want_b = getattr(Run(precision, M, B), between)()
    r = Run(precision, M, A)
    for _ in range(4):
        r.forward()
    assert r.ctx.paths() & GRAPH
    atomics = precision == "fp64" and between == "adjoint"
    for _ in range(2):
        r.ctx.set_box(*B)
        assert same(getattr(r, between)(), want_b, atomics)
        r.ctx.set_box(*A)
        r.f.zero_()
        assert torch.equal(r.forward(), want)
    assert not same(getattr(r, between)(), want_b, atomics)


@pytest.mark.parametrize("precision,M", GRIDS)
def test_replay_among_gradients_and_virials(precision, M):
    box = (1.0 * M,) * 3
    names = ["forward", "virial_after_forward", "adjoint", "forward", "separate", "forward",
             "adjoint", "virial", "forward", "virial_after_forward"]
    want = {k: getattr(Run(precision, M, box), k)() for k in ("forward", "adjoint", "virial",
                                                              "separate")}
    fresh = Run(precision, M, box)
    fresh.forward()
    want["virial_after_forward"] = fresh.virial_after_forward()
    r = Run(precision, M, box)
    for _ in range(4):
        r.forward()
    assert r.ctx.paths() & GRAPH
    assert bool(r.ctx.paths() & OWN_FFT) == (precision == "mixed" and M == 64)
    for k in names:
        r.f.zero_()
        assert same(getattr(r, k)(), want[k], precision == "fp64" and k == "adjoint"), k
    assert r.ctx.paths() & GRAPH
