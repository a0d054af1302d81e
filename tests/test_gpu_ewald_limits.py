"""Ewald reciprocal sums with large and small cut-offs at the same time: the force
kernel's shared memory grows with the cut-off, and the limit that a thread sets for it
holds for every thread of the process.  Every call succeeds and gives what it gives
alone, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kcuts", [(3, 62), (64, 120)])
def test_threads_with_unequal_cutoffs(kcuts):
    import torch
    from gse_b200.gse import ewald_recip
    rng = np.random.default_rng(1)
    x = rng.uniform(0.0, 10.0, (40, 4))
    x[:, 3] = np.where(np.arange(40) % 2, 1.0, -1.0)
    box = (10.0, 10.0, 10.0)

    def call(kcut, stream):
        return ewald_recip(0.2, kcut, box, x, stream=stream)

    want = {k: call(k, None) for k in kcuts}
    failed = []

    def work(kcut, repeats):
        stream = torch.cuda.Stream()
        try:
            for _ in range(repeats):
                e, f = call(kcut, stream.cuda_stream)
                assert e == want[kcut][0] and np.array_equal(f, want[kcut][1])
        except Exception as err:  # reported by the test's own thread
            failed.append(err)

    threads = [threading.Thread(target=work, args=(k, 400 if k == kcuts[0] else 150))
               for k in kcuts for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
