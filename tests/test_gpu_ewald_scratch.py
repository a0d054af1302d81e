"""The Ewald reciprocal sum in pieces: rows that go in several blocks (from a cut-off of
about 120 on), and a device that is short of memory, where both rows and atoms go in
smaller pieces instead of failing.  Against the oracle within the tolerance of the
sum's other tests (1e-12), with a width that leaves the terms at the cut-off at e^-2 of
the first; a phase at kcut 255 carries 2 pi 255 2^-53 = 2e-13, twice in a force term.
The oracle's phases come from whole angles of some 3000, at kcut 255 they leave 2e-12
in its forces (by the same sum in 80 bits): there the sum is written out, with phases of
reduced angles in 80 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX = (11.0, 13.5, 9.25)


def system(n, charged):
    rng = np.random.default_rng(n)
    x = np.zeros((n, 4))
    x[:, :3] = rng.uniform(-0.5, 1.5, (n, 3)) * np.array(BOX)
    at = np.concatenate([[0, n - 1], rng.choice(np.arange(1, n - 1), charged - 2, replace=False)])
    x[at, 3] = rng.uniform(0.5, 1.5, charged) * np.where(np.arange(charged) % 2, 1.0, -1.0)
    return x


def written_out(sigma, kcut, box, x, ccelec=332.0716):
    k = np.arange(-kcut, kcut + 1)
    phase = []
    for d in range(3):
        t = np.outer(k.astype(np.longdouble), x[:, d].astype(np.longdouble) / box[d])
        a = 2 * np.arccos(np.longdouble(-1)) * (t - np.rint(t))
        phase.append((np.cos(a) + 1j * np.sin(a)).astype(np.complex128))
    kv = [2 * np.pi * k / b for b in box]
    q, E, F = x[:, 3], 0.0, np.zeros((len(x), 3))
    for kz in range(kcut + 1):
        i = kz + kcut
        on = (k[:, None] ** 2 + k ** 2 + kz * kz <= kcut * kcut)  # [ky, kx]
        if kz == 0:
            on &= (k[:, None] > 0) | ((k[:, None] == 0) & (k > 0))
        k2 = np.where(on, kv[1][:, None] ** 2 + kv[0] ** 2 + kv[2][i] ** 2, 1.0)
        P = np.where(on, 2 * np.pi / np.prod(box) * ccelec * np.exp(-0.5 * sigma ** 2 * k2) / k2, 0)
        r = phase[1] * phase[2][i]  # [ky, atom]
        S = (r * q) @ phase[0].T
        E += 2 * (P * np.abs(S) ** 2).sum()
        U = P * np.conj(S)
        g, gx = (U @ phase[0] * r).imag, ((U * kv[0]) @ phase[0] * r).imag
        F += 4 * q[:, None] * np.stack([gx.sum(0), kv[1] @ g, kv[2][i] * g.sum(0)], axis=1)
    return E, F


def check(n, charged, kcut):
    import oracle
    from gse_b200.gse import ewald_recip
    x = system(n, charged)
    sigma = 2.0 / (2.0 * np.pi * kcut / max(BOX))
    E, F = ewald_recip(sigma, kcut, BOX, x)
    on = x[:, 3] != 0.0
    reference = written_out if kcut == 255 else oracle.ewald_recip
    E0, F0 = reference(sigma, kcut, BOX, np.ascontiguousarray(x[on]))
    assert abs(E - E0) <= 1e-12 * abs(E0)
    d = np.sqrt(((F[on] - F0) ** 2).sum() / (F0 ** 2).sum())
    assert d <= 1e-12, d
    assert not F[~on].any()
    assert abs(ewald_recip(sigma, kcut, BOX, x, forces=False)[0] - E) <= 1e-13 * abs(E)


@pytest.mark.parametrize("n,charged,kcut", [(130, 16, 119), (130, 16, 121), (66, 8, 160),
                                            (5, 4, 255)])
def test_rows_in_blocks(n, charged, kcut):
    check(n, charged, kcut)


@pytest.mark.parametrize("left_mb,n,charged,kcut", [
    (450, 5, 4, 255),       # the rows' sums of one block alone would take 2.4 GB
    (60, 100001, 32, 60),   # the phase tables alone 293 MB
    (24, 3000, 16, 90),     # 80 MB of rows' sums, 13 MB of tables
])
def test_short_device(left_mb, n, charged, kcut):
    import torch
    check(70, 4, 70)  # every kernel is loaded before the memory is taken
    check(70, 4, 5)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    taken = torch.empty(free - (left_mb << 20), dtype=torch.uint8, device="cuda")
    try:
        check(n, charged, kcut)
    finally:
        del taken
        torch.cuda.empty_cache()
