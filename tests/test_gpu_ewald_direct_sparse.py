"""The Ewald direct sum in boxes with far more cells than atoms: against the oracle (1e-12
of the forces' RMS and of the energy, as in the sum's other tests), the same bits on
every run, and at a cost that goes with the atoms, not with the empty cells (a block for
each of 1.4 million cells made it 60 times the same atoms' cost in a smaller box; ten
times is allowed here)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def system(n, box, drop):
    rng = np.random.default_rng(n)
    x = np.empty((n, 4))
    if drop:  # everything in one corner of the box, some atoms on the other side of it
        i = np.arange(n)
        x[:, :3] = 1.1 * np.stack([i % 16, i // 16 % 16, i // 256], axis=1)
        x[:, :3] += rng.uniform(-0.3, 0.3, (n, 3))
    else:
        x[:, :3] = rng.uniform(0.0, 1.0, (n, 3)) * np.array(box)
    x[:, 3] = rng.uniform(0.5, 1.5, n) * np.where(np.arange(n) % 2, 1.0, -1.0)
    return x


@pytest.mark.parametrize("n,box,rcut,drop", [
    (1, (50.0, 50.0, 50.0), 0.5, False),
    (2, (50.0, 60.0, 70.0), 0.7, True),
    (1000, (100.0, 90.0, 80.0), 4.0, False),
    (1500, (200.0, 150.0, 180.0), 2.5, True),
    (3000, (40.0, 400.0, 30.0), 5.0, True),
])
def test_mostly_empty_cells(n, box, rcut, drop):
    import oracle
    from gse_b200 import workloads as W
    from gse_b200.gse import ewald_direct
    x = system(n, box, drop)
    ib, nb = W.triplet_exclusions(n)
    e0, f0 = oracle.ewald_direct(3.0, rcut, box, x, iblo14=ib, inb14=nb)
    e, f = ewald_direct(3.0, rcut, box, x, ib, nb)
    assert abs(e - e0) <= 1e-12 * abs(e0)
    assert np.sqrt(((f - f0) ** 2).sum()) <= 1e-12 * np.sqrt((f0 ** 2).sum())
    for _ in range(5):
        e1, f1 = ewald_direct(3.0, rcut, box, x, ib, nb)
        assert e1 == e and np.array_equal(f1, f)


def test_cost_of_empty_cells():
    from gse_b200.gse import ewald_direct
    x = system(1000, (1.0, 1.0, 1.0), False)

    def cost(L, rcut):
        y = x * np.array([L, L, L, 1.0])
        best = np.inf
        for _ in range(20):
            t = time.perf_counter()
            ewald_direct(2.0, rcut, (L, L, L), y)
            best = min(best, time.perf_counter() - t)
        return best

    assert cost(100.0, 0.9) <= 10 * cost(30.0, 3.0)
