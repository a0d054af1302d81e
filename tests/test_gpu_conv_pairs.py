"""The on-grid convolution's packed FP32 passes against the oracle, bit for bit, where
their pairing ends: odd and even row lengths and row counts, runs longer than a warp's
160 outputs and a block's 80, axes shorter than the taps, and grids whose start is
aligned to 4 bytes only (which the paired y and z passes do not take)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [0.9, 1.85])  # 9 and 17 taps at h = 1
@pytest.mark.parametrize("M,offset", [
    ((16, 16, 16), 0), ((16, 16, 16), 1), ((17, 15, 13), 0), ((34, 3, 5), 0), ((6, 81, 7), 0),
    ((162, 9, 82), 0), ((161, 8, 80), 0), ((2, 160, 2), 2), ((322, 5, 3), 3),
])
def test_paired_passes_equal_oracle(M, offset, sigma):
    import oracle
    import torch
    from gse_b200.gse import Context
    box = tuple(float(m) for m in M)
    rcut = 3.0 * np.sqrt(2.0) * sigma
    rho = np.random.default_rng(M[0]).standard_normal((M[2], M[1], M[0])).astype(np.float32)
    want = oracle.spread_on_grid(M, box, sigma, rcut, rho, dtype=np.float32)
    ctx = Context(*M, sigma=1.0, boxx=box[0], boxy=box[1], boxz=box[2], precision="mixed")
    size = rho.size
    bufs = [torch.zeros(size + 4, dtype=torch.float32, device="cuda") for _ in range(2)]
    a, o = (b[offset:offset + size] for b in bufs)
    a.copy_(torch.from_numpy(rho.reshape(-1)))
    ctx.gauss_spread_on_grid(sigma, rcut, *box, a, o)
    torch.cuda.synchronize()
    assert np.array_equal(o.cpu().numpy().reshape(-1), np.asarray(want).reshape(-1))
