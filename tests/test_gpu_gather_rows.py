"""The gather's row list and brick shapes against the oracle: every stencil width, grids
that take each of the three brick shapes in either form, spacings that differ between
the axes (the rows within reach then are an ellipse), and FP32 coordinates so large
that their rounding moves an atom away from its stencil centre.

Tolerance, of the sum of the terms' magnitudes: FP64 some 30 roundings in a row's and a
lane's sums (1e-14 with room); mixed 1e-6 for the hardware exponential plus about 25
FP32 roundings (2e-6)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGMA1 = 2.0 * np.sqrt(0.4)
RCUT = 3.0 * np.sqrt(2.0) * SIGMA1


def magnitudes(M, box, x, phi):
    """Sum over the sphere of |q pref e phi d| per atom and axis, in FP64."""
    h = [b / m for b, m in zip(box, M)]
    out = np.zeros((x.shape[0], 3))
    pref = (2 * np.pi) ** -1.5 * np.prod(h) * SIGMA1 ** -5
    for i, a in enumerate(x):
        idx, d = [], []
        for k in range(3):
            n = int(np.ceil(RCUT / h[k]))
            t = np.arange(-n, n + 1) + int(np.round(a[k] / h[k]))
            idx.append(np.mod(t, M[k]))
            d.append(a[k] - t * h[k])
        r2 = d[2][:, None, None] ** 2 + d[1][None, :, None] ** 2 + d[0][None, None, :] ** 2
        w = np.where(r2 < RCUT ** 2 * 1.01, np.exp(-r2 / (2 * SIGMA1 ** 2)), 0.0)
        w = w * np.abs(phi[np.ix_(idx[2], idx[1], idx[0])]) * pref * abs(a[3])
        out[i] = [(w * np.abs(d[0])[None, None, :]).sum(), (w * np.abs(d[1])[None, :, None]).sum(),
                  (w * np.abs(d[2])[:, None, None]).sum()]
    return out


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-14), ("mixed", 3e-6)])
@pytest.mark.parametrize("M,h,shift", [
    ((20, 20, 20), (0.95, 0.95, 0.95), 0),   # 16 x 8 x 4 bricks
    ((39, 21, 30), (0.92, 1.0, 1.07), 0),
    ((33, 40, 41), (0.78, 0.82, 0.88), 0),   # width 15
    ((64, 64, 64), (1.1, 1.3, 1.2), 0),      # width 11; mixed 16 x 8 x 8
    ((64, 50, 64), (1.35, 1.5, 1.7), 0),     # width 9
    ((80, 80, 100), (0.95, 1.05, 1.0), 0),   # 16 x 16 x 8
    ((20, 20, 20), (1.0, 1.0, 1.0), 20000),  # |x| = 4e5: FP32 spacing 1/32
])
def test_gather_equals_oracle(M, h, shift, precision, tol):
    import oracle
    from gse_b200.gse import CpuGaussCharge, CpuGrid
    dt = np.float64 if precision == "fp64" else np.float32
    n, box = 150, tuple(a * b for a, b in zip(h, M))
    rng = np.random.default_rng(M[1])
    x = np.empty((n, 4), dtype=dt)
    x[:, :3] = (rng.uniform(-0.5, 1.5, (n, 3)) + shift) * np.array(box)
    x[:, 3] = rng.standard_normal(n)
    phi = CpuGrid(*M, dt)
    phi.data[...] = rng.standard_normal(phi.data.shape)
    f = [np.zeros(n) for _ in range(3)]
    CpuGaussCharge(*M, precision=precision).interpolateForce(SIGMA1, RCUT, n, x, *box, phi, *f)
    want = np.asarray(oracle.gather(M, box, SIGMA1, RCUT, x, phi.data, dtype=dt))
    want = want if want.shape == (n, 3) else want.T
    scale = magnitudes(M, box, x.astype(np.float64), phi.data.astype(np.float64))
    assert np.all(np.abs(np.stack(f, 1) - want) <= tol * scale)
