"""The Ewald reciprocal sum against the oracle at the edges of its tiles: atom counts
around the 32- and 64-atom tiles, k cut-offs around the 8-column strips, the
80-column tile, the 32-entry chunks and the switch to 32-atom force blocks
(kcut 63/64), boxes of unequal sides, and more atoms than one slab of phase
tables holds.

Tolerance: a phase 2 pi k x / L carries about 2 pi kcut 2^-53 of error on either
side (5e-14 at kcut 66), which a term of the energy or the forces takes on once or
twice; 1e-12 of the forces' RMS and of the energy covers sums of such terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(box, x, kcut, sigma):
    import oracle
    from gse_b200.gse import ewald_recip
    E, F = ewald_recip(sigma, kcut, box, x)
    on = x[:, 3] != 0.0
    E0, F0 = oracle.ewald_recip(sigma, kcut, box, np.ascontiguousarray(x[on]))
    assert abs(E - E0) <= 1e-12 * abs(E0)
    d = np.sqrt(((F[on] - F0) ** 2).sum() / (F0 ** 2).sum())
    assert d <= 1e-12, d
    assert not F[~on].any()
    assert ewald_recip(sigma, kcut, box, x, forces=False)[0] == E


@pytest.mark.parametrize("n,kcut", [(2, 1), (31, 3), (32, 4), (33, 39), (63, 40), (64, 15),
                                    (65, 16), (129, 63), (70, 64), (40, 66)])
def test_tile_edges(n, kcut):
    rng = np.random.default_rng(1000 * n + kcut)
    box = (11.0, 13.5, 9.25)
    x = np.empty((n, 4))
    x[:, :3] = rng.uniform(-0.5, 1.5, (n, 3)) * np.array(box)
    x[:, 3] = rng.uniform(0.5, 1.5, n) * np.where(np.arange(n) % 2, 1.0, -1.0)
    # a width that leaves the terms at the cut-off at e^-2 of the first ones
    check(box, x, kcut, 2.0 / (2.0 * np.pi * kcut / max(box)))


def test_more_atoms_than_one_slab():
    n, kcut, box = 100001, 60, (20.0, 20.0, 20.0)
    rng = np.random.default_rng(5)
    x = np.zeros((n, 4))
    x[:, :3] = rng.uniform(0.0, 20.0, (n, 3))
    at = np.concatenate([[0, n - 1], rng.choice(np.arange(1, n - 1), 62, replace=False)])
    x[at, 3] = rng.standard_normal(64)
    check(box, x, kcut, 2.0 / (2.0 * np.pi * kcut / 20.0))
