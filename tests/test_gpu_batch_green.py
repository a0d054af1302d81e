"""Batch energies where several systems share one block's run of spectrum bins: many
systems of the smallest grid, larger and odd-sided ones between them.

Tolerance: that of the batch's other comparison with single-system contexts (energies
within 1e-6: the grids' rounding, and the weights' in the same arithmetic), since the
product with G and the energy terms are formed as there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_energies_of_systems_within_one_run():
    from gse_b200 import workloads as W
    from gse_b200.gse import Batch, Context
    sides = ([(10, 10, 10)] * 5 + [(11, 13, 10)] * 3 + [(20, 18, 16)] + [(10, 10, 10)] * 4
             + [(30, 11, 12)])
    desc, xs = [], []
    for k, M in enumerate(sides):
        n, box = 60 + 9 * k, tuple(0.98 * m for m in M)
        scale = np.array([box[0], box[1], box[2], 10.0]) / 10.0
        desc.append({"size": M, "box": box, "n": n})
        xs.append((W.triplets(n, 10.0, k) * scale).astype(np.float32))
    E, _ = Batch(desc, sigma=2.0, kappa=0.4, lambdaSigma1=3.0).forward(np.concatenate(xs))
    for k, (d, x) in enumerate(zip(desc, xs)):
        ctx = Context(*d["size"], 2.0, 0.4, 3.0, 3.0, *d["box"], precision="mixed")
        want = ctx.forward(d["n"], x, *(np.zeros(d["n"]) for _ in range(3)))
        assert abs(E[k] - want) <= 1e-6 * abs(want), k
