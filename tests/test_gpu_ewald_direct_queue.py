"""The Ewald direct sum's pair queues: every number of entries that a drain of 32 can
leave behind (one to 32 partners are found a step, at every density from a few to all
of the staged atoms), against the oracle and, as each atom's terms are summed in a
fixed order, the same bits on every run.  A partner lost or taken twice moves a force
by far more than the tolerance of the direct sum's other tests, 1e-12 of the RMS."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rcut", [3.0, 4.5, 6.0, 8.0, 11.0])
def test_drains_keep_every_partner(rcut):
    import oracle
    from gse_b200.gse import ewald_direct
    n, box = 1500, (20.0, 21.0, 22.0)
    rng = np.random.default_rng(int(10 * rcut))
    x = np.empty((n, 4))
    i = rng.permutation(12 ** 3)[:n]  # a shaken lattice: no pair is close, none outweighs the rest
    cell = np.stack([i % 12, i // 12 % 12, i // 144], axis=1) + rng.uniform(-0.3, 0.3, (n, 3))
    x[:, :3] = cell / 12.0 * np.array(box)
    x[:, 3] = rng.uniform(0.5, 1.5, n) * np.where(np.arange(n) % 2, 1.0, -1.0)
    e0, f0 = oracle.ewald_direct(6.0, rcut, box, x)
    e, f = ewald_direct(6.0, rcut, box, x)
    assert abs(e - e0) <= 1e-12 * abs(e0)
    assert np.sqrt(((f - f0) ** 2).sum()) <= 1e-12 * np.sqrt((f0 ** 2).sum())
    for _ in range(10):
        e1, f1 = ewald_direct(6.0, rcut, box, x)
        assert e1 == e and np.array_equal(f1, f)
