"""The Ewald direct sum against the oracle where its blocks and tiles end: cells far
fuller than the mean (several rounds of 32 atoms per block), more neighbours than
one staged tile (3072), atom counts around a block's 32 and a warp's 2, cut-offs
that nearly nobody and nearly everybody meets.

Tolerance: a pair term carries some ten roundings (1e-15 of its size), an atom sums
up to 4000 of them in another order than the oracle (at most 4000 x 2^-53 of the
sum of the sizes, in practice its root); 1e-12 of the forces' RMS and of the energy
as in the other tests of this sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box,rcut,cluster", [
    (1, (20.0, 20.0, 20.0), 5.0, 0.0),
    (31, (20.0, 21.0, 22.0), 5.0, 0.0),
    (33, (9.0, 9.0, 9.0), 4.4, 0.0),
    (65, (30.0, 12.0, 9.5), 9.0, 0.0),
    (700, (60.0, 60.0, 60.0), 1.5, 0.0),
    (3500, (60.0, 60.0, 60.0), 6.0, 0.9),   # most atoms in a corner cell
    (4000, (25.0, 25.0, 25.0), 12.0, 0.0),  # eight cells, all of them neighbours
])
def test_block_and_tile_edges(n, box, rcut, cluster):
    import oracle
    from gse_b200 import workloads as W
    from gse_b200.gse import ewald_direct
    rng = np.random.default_rng(n)
    x = np.empty((n, 4))
    x[:, :3] = rng.uniform(0.0, 1.0, (n, 3)) * np.array(box)
    m = int(cluster * n)
    x[:m, :3] = rng.uniform(0.0, 1.0, (m, 3)) * 5.0
    x[:, 3] = rng.uniform(0.5, 1.5, n) * np.where(np.arange(n) % 2, 1.0, -1.0)
    ib, nb = W.triplet_exclusions(n)
    e0, f0 = oracle.ewald_direct(2.0, rcut, box, x, iblo14=ib, inb14=nb)
    e, f = ewald_direct(2.0, rcut, box, x, ib, nb)
    assert abs(e - e0) <= 1e-12 * abs(e0)
    scale = np.sqrt((f0 ** 2).sum())
    assert np.sqrt(((f - f0) ** 2).sum()) <= 1e-12 * scale
