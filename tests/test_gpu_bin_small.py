"""The one-launch binning of few atoms at the ends of its range (512 atoms in FP64, 1024
in mixed, 10240 bins) and just past them, with atoms spread out and all in one bin.

FP64: against the oracle's spread, within 1e-13 of the sum of the terms' magnitudes as
in the spread's own test, and the same bits on each run (the order in a bin).  Mixed:
its integer sums do not depend on the order of the atoms, and atoms of no charge change
neither them nor the scale, so with such atoms added until the general binning takes
the call the grid is the same bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGMA1 = 2.0 * np.sqrt(0.4)
RCUT = 3.0 * np.sqrt(2.0) * SIGMA1
GRIDS = [(20, 20, 20), (40, 32, 32), (41, 32, 32), (160, 32, 32)]


def atoms(n, box, dt, crowded):
    rng = np.random.default_rng(n + int(box[0]))
    x = np.empty((n, 4), dtype=dt)
    x[:, :3] = (0.475 + 0.3 * rng.uniform(-1, 1, (n, 3)) if crowded
                else rng.uniform(-0.2, 1.2, (n, 3)) * np.array(box))
    x[:, 3] = rng.standard_normal(n)
    return x


def spread(precision, M, box, x):
    from gse_b200.gse import CpuGaussCharge, CpuGrid
    rho = CpuGrid(*M, x.dtype.type)
    CpuGaussCharge(*M, precision=precision).spreadChargeToGrid(
        SIGMA1, RCUT, x.shape[0], x, *box, rho)
    return np.array(rho.data)


@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("M", GRIDS[:3])
@pytest.mark.parametrize("n", [1, 512, 513])
def test_small_fp64_binning_equals_oracle(n, M, crowded):
    import oracle
    box = tuple(0.95 * m for m in M)
    x = atoms(n, box, np.float64, crowded)
    got = spread("fp64", M, box, x)
    assert np.array_equal(got, spread("fp64", M, box, x))
    want = oracle.spread(M, box, SIGMA1, RCUT, x).reshape(got.shape)
    x[:, 3] = np.abs(x[:, 3])
    scale = oracle.spread(M, box, SIGMA1, RCUT, x).reshape(got.shape)
    assert np.all(np.abs(got - want) <= 1e-13 * scale + 1e-300)


@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("M", GRIDS)
@pytest.mark.parametrize("n", [1, 1024])
def test_small_mixed_binning_equals_general(n, M, crowded):
    box = tuple(0.95 * m for m in M)
    x = atoms(n, box, np.float32, crowded)
    more = atoms(1025 - n, box, np.float32, not crowded)
    more[:, 3] = 0
    assert np.array_equal(spread("mixed", M, box, x),
                          spread("mixed", M, box, np.concatenate([x, more])))
