"""The FP64 tiled spread against the oracle, at the sizes where its tiling can go
wrong: the smallest grid (regions that wrap several times), sides that are not
multiples of the 8-point patches, every block shape of the launch rule, every
stencil width, atom counts around the chunk and list sizes.

Tolerance: a weight is a product of three 1-D weights, each formed by about a
dozen roundings from exponentials of arguments below 10 (some 50 ulp in all,
1e-14), and a point sums at most a few thousand terms; 1e-13 of the sum of the
terms' magnitudes covers both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGMA1 = 2.0 * np.sqrt(0.4)
RCUT = 3.0 * np.sqrt(2.0) * SIGMA1


@pytest.mark.parametrize("M,h,n", [
    ((10, 10, 10), 0.95, 65),       # three periods of the grid reach one block
    ((11, 10, 13), 1.0, 1),
    ((20, 20, 20), 0.95, 6000),     # more atoms than one list holds
    ((17, 23, 31), 0.85, 64),       # width 15
    ((33, 40, 31), 1.15, 63),       # width 11
    ((41, 33, 27), 1.4, 3001),      # width 9
    ((64, 57, 60), 0.95, 2048),     # blocks of 1 x 1 x 2 patches
    ((80, 73, 80), 0.95, 2049),     # 1 x 2 x 2 patches
    ((96, 90, 100), 0.95, 5000),    # 1 x 1 x 2 patches again
    ((144, 128, 136), 0.8, 5000),   # 2 x 2 x 2 patches, width 15
    ((144, 128, 136), 1.35, 5000),  # 2 x 2 x 2 patches, width 9
])
def test_fp64_spread_equals_oracle(M, h, n):
    import oracle
    from gse_b200.gse import CpuGaussCharge, CpuGrid
    box = tuple(h * m for m in M)
    rng = np.random.default_rng(n)
    x = np.empty((n, 4))
    x[:, :3] = rng.uniform(-0.2, 1.2, (n, 3)) * np.array(box)
    x[:, 3] = rng.standard_normal(n)
    rho = CpuGrid(*M)
    CpuGaussCharge(*M, precision="fp64").spreadChargeToGrid(SIGMA1, RCUT, n, x, *box, rho)
    want = oracle.spread(M, box, SIGMA1, RCUT, x)
    x[:, 3] = np.abs(x[:, 3])
    scale = oracle.spread(M, box, SIGMA1, RCUT, x)
    assert np.all(np.abs(rho.data - want.reshape(rho.data.shape))
                  <= 1e-13 * scale.reshape(rho.data.shape) + 1e-300)
