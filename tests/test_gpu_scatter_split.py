"""The mixed spread's bricks whole and split over several blocks, on the grids where the
number of blocks per brick changes (at width 15, whose blocks have an SM each, another
grid than at 13), with charges spread out, few, and crowded into one corner: the density
against the oracle's within 1e-5 of the largest value (as in the spread's stage tests),
and, as its sums are integer, the same bits for any order of the atoms, which goes with
which block takes an atom."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGMA1 = 2.0 * np.sqrt(0.4)
RCUT = 3.0 * np.sqrt(2.0) * SIGMA1


@pytest.mark.parametrize("M", [(48, 64, 64), (64, 64, 64), (64, 76, 64), (80, 80, 80), (96, 90, 108)])
@pytest.mark.parametrize("h", [0.82, 0.97])
def test_density(M, h):
    import oracle
    from gse_b200.gse import CpuGaussCharge, CpuGrid
    box = tuple(h * m for m in M)
    gauss = CpuGaussCharge(*M, precision="mixed")
    for n, crowded in ((40, False), (1500, False), (1500, True)):
        rng = np.random.default_rng(n)
        x = np.empty((n, 4), dtype=np.float32)
        x[:, :3] = rng.uniform(-0.1, 1.1, (n, 3)) * np.array(box) * (0.2 if crowded else 1.0)
        x[:, 3] = rng.uniform(0.5, 1.0, n) * np.where(np.arange(n) % 2, 1.0, -1.0)
        rho = []
        for order in (np.arange(n), rng.permutation(n)):
            g = CpuGrid(*M, np.float32)
            gauss.spreadChargeToGrid(SIGMA1, RCUT, n, np.ascontiguousarray(x[order]), *box, g)
            rho.append(np.array(g.data).reshape(M[::-1]).copy())
        assert np.array_equal(rho[0], rho[1])
        want = oracle.spread(M, box, SIGMA1, RCUT, x.astype(np.float64)).reshape(M[::-1])
        assert np.abs(rho[0] - want).max() <= 1e-5 * np.abs(want).max()
