"""The Ewald calls' scratch pool under several threads and streams: overlapping calls of
different sizes give what the same calls give one after the other, bit for bit (their
sums run in a fixed order)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_overlapping_calls_equal_serial_ones():
    import torch
    from gse_b200 import workloads as W
    from gse_b200.gse import ewald_direct, ewald_recip
    jobs = [(300 * (k + 1), 12.0 + 4.0 * k, 6 + 5 * k) for k in range(4)]
    xs = [W.triplets(n, L, n).astype(np.float64) for n, L, _ in jobs]

    def call(k, stream):
        n, L, kcut = jobs[k]
        box = (L, L, L)
        e1, f1 = ewald_recip(2.0, kcut, box, xs[k], stream=stream)
        e2, f2 = ewald_direct(2.0, 0.45 * L, box, xs[k], *W.triplet_exclusions(n), stream=stream)
        return e1, e2, f1, f2

    want = [call(k, None) for k in range(4)]
    streams = [torch.cuda.Stream() for _ in range(4)]
    got, failed = {}, []

    def work(k):
        try:
            for r in range(8):
                got[k, r] = call(k, streams[k].cuda_stream)
        except Exception as e:  # reported by the test's own thread
            failed.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for (k, _), g in got.items():
        assert g[0] == want[k][0] and g[1] == want[k][1]
        assert np.array_equal(g[2], want[k][2]) and np.array_equal(g[3], want[k][3])
