"""The gradient's kernels against the same derivatives written out in numpy (FP64), at
the shapes where they change: the FP64 form and the mixed form's tiled and
atom-parallel kernels, stencils of unequal widths per axis, wider than a half-warp's
16 offsets, wider than the grid, with and without force cotangents.

Tolerance, of each gradient's largest component: FP64 the FFT's and the sums' rounding
(1e-12 as in the other FP64 tests); mixed 2e-5 (FP32 grids and transforms, whose
rounding 1e-7 of the largest grid value meets cancelling sums of alternating charges)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CCELEC = 332.0716


def gradient(M, box, sigma, x, dE, G):
    """(dL/dq, dL/dx, dL/dy, dL/dz) of L = dE E + sum G . F, plain numpy."""
    h = np.array(box) / np.array(M)
    s1, s2 = sigma * np.sqrt(0.4), sigma * np.sqrt(0.2)
    rcut = 3.0 * np.sqrt(2.0) * s1
    pref = (2 * np.pi * s1 ** 2) ** -1.5
    cA = CCELEC * (2 * np.pi) ** -1.5 * np.prod(h) * s1 ** -5

    def stencil(a):
        idx, u = [], []
        for k in range(3):
            n = int(np.ceil(rcut / h[k]))
            p = a[k] / h[k]
            t = np.arange(-n, n + 1) + int(np.sign(p) * np.floor(abs(p) + 0.5))
            idx.append(np.mod(t, M[k]))
            u.append(a[k] - t * h[k])
        at = np.ix_(idx[2], idx[1], idx[0])
        u = (u[0][None, None, :], u[1][None, :, None], u[2][:, None, None])
        r2 = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        return at, u, np.exp(-r2 / (2 * s1 ** 2)), r2 < rcut ** 2

    k = [2 * np.pi * np.fft.fftfreq(m, 1.0 / m) / b for m, b in zip(M, box)]
    k2 = k[0][None, None, :] ** 2 + k[1][None, :, None] ** 2 + k[2][:, None, None] ** 2
    k2[0, 0, 0] = 1.0
    green = 4 * np.pi * np.exp(-0.5 * s2 ** 2 * k2) / k2
    green[0, 0, 0] = 0.0

    def solve(rho):
        return np.fft.ifftn(np.fft.fftn(rho) * green).real

    rho, lam = np.zeros(M[::-1]), np.zeros(M[::-1])
    for a, g in zip(x, G):
        at, u, e, ball = stencil(a)
        np.add.at(rho, at, a[3] * pref * e)
        np.add.at(lam, at, cA * a[3] * np.where(ball, e, 0.0) * sum(g[d] * u[d] for d in range(3)))
    phi = solve(rho)
    psi = solve(lam) + dE * CCELEC * np.prod(h) * phi
    out = np.zeros((4, len(x)))
    for i, (a, g) in enumerate(zip(x, G)):
        at, u, e, ball = stencil(a)
        c, t = pref * e * psi[at], cA * np.where(ball, e, 0.0) * phi[at]
        gu = sum(g[d] * u[d] for d in range(3))
        out[0, i] = (c + t * gu).sum()
        for d in range(3):
            out[1 + d, i] = a[3] * (-(c + t * gu) * u[d] / s1 ** 2 + t * g[d]).sum()
    return out


@pytest.mark.parametrize("cotangents", [True, False])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 2e-5)])
@pytest.mark.parametrize("M,h", [
    ((20, 20, 20), (0.95, 0.95, 0.95)),   # width 13, tiled in the mixed form
    ((16, 24, 17), (1.1, 1.2, 1.15)),     # width 11, odd side
    ((24, 20, 22), (0.7, 1.0, 1.4)),      # 17 x 13 x 9: atom-parallel in both forms
    ((9, 12, 11), (1.0, 0.6, 0.9)),       # wider than the grid on two axes
    ((40, 12, 10), (0.3, 1.3, 2.0)),      # 37 x offsets: three runs
])
def test_gradient_equals_written_out(M, h, precision, tol, cotangents):
    from gse_b200.gse import Context
    box = tuple(a * b for a, b in zip(M, h))
    n, sigma = 37, 2.0
    rng = np.random.default_rng(M[0])
    x = np.empty((n, 4))
    x[:, :3] = rng.uniform(-0.3, 1.3, (n, 3)) * np.array(box)
    x[:, 3] = rng.uniform(0.5, 1.0, n) * np.where(np.arange(n) % 2, 1.0, -1.0)
    x = x.astype(np.float32).astype(np.float64)
    G = rng.standard_normal((n, 3)) if cotangents else np.zeros((n, 3))
    want = gradient(M, box, sigma, x, 0.7, G)
    ctx = Context(*M, sigma, 0.4, 3.0, 3.0, *box, precision=precision)
    xin = np.ascontiguousarray(x, dtype=ctx.dtype)
    got = [np.zeros(n) for _ in range(4)]
    g = [np.ascontiguousarray(G[:, d]) if cotangents else None for d in range(3)]
    ctx.adjoint(n, xin, 0.7, *g, *got)
    for a, b in zip(got, want):
        assert np.abs(a - b).max() <= tol * np.abs(want[0 if b is want[0] else slice(1, 4)]).max()
