"""Few atoms on large grids: the binning writes every bin whatever the number of atoms.
The density against the oracle's within 1e-13 (FP64, as in the spread's own test) and
1e-5 of the largest value (mixed, as in its stage tests), call after call with other
atoms (the counts are zero again), and a cost that does not fall with more atoms: a
placement sized by the atoms alone made 30 of them dearer than 20,000."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGMA1 = 2.0 * np.sqrt(0.4)
RCUT = 3.0 * np.sqrt(2.0) * SIGMA1


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_density_of_few_atoms(precision):
    import oracle
    from gse_b200.gse import CpuGaussCharge, CpuGrid
    M = (100, 66, 57)
    box = tuple(0.97 * m for m in M)
    dt = np.float64 if precision == "fp64" else np.float32
    gauss = CpuGaussCharge(*M, precision=precision)
    for n in (30, 1, 700, 257, 1500):
        rng = np.random.default_rng(n)
        x = np.empty((n, 4), dtype=dt)
        x[:, :3] = rng.uniform(-0.2, 1.2, (n, 3)) * np.array(box)
        x[:, 3] = rng.uniform(0.5, 1.0, n)
        rho = CpuGrid(*M, dt)
        gauss.spreadChargeToGrid(SIGMA1, RCUT, n, x, *box, rho)
        want = oracle.spread(M, box, SIGMA1, RCUT, x.astype(np.float64))
        got = np.array(rho.data).reshape(want.shape)
        if precision == "fp64":
            assert np.all(np.abs(got - want) <= 1e-13 * want + 1e-300)
        else:
            assert np.abs(got - want).max() <= 1e-5 * want.max()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_few_atoms_cost_no_more_than_many(precision):
    import torch
    from gse_b200 import workloads as W
    from gse_b200.gse import Context
    M, L = 144, 140.0
    ctx = Context(M, M, M, 2.0, 0.4, 3.0, 3.0, L, L, L, precision=precision)
    dt = torch.float64 if precision == "fp64" else torch.float32

    def cost(n):
        x = torch.from_numpy(W.triplets(n, L, 1)).to(dt).cuda()
        f = torch.zeros(3, n, dtype=torch.float64, device="cuda")
        best = np.inf
        ctx.spread_charge(n, x)
        ctx.solve_poisson()
        for _ in range(30):
            torch.cuda.synchronize()
            t = time.perf_counter()
            ctx.interpolate_force(n, x, f[0], f[1], f[2])
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        return best

    many = cost(20001)
    assert cost(30) <= many
    assert cost(1500) <= many
