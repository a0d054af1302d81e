"""The electric field on the grid at row lengths around a lane's four and five positions
per step, and beside the wrap: the same bits as numpy's separately rounded differences
and products in the form's own type."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("mx", [12, 32, 127, 128, 129, 149, 150, 160, 161, 256, 257, 300, 320, 321])
def test_rows(mx, precision):
    import torch
    from gse_b200.gse import Context
    dt = np.float64 if precision == "fp64" else np.float32
    M, box = (mx, 11, 13), (0.9 * mx, 10.5, 13.5)
    ctx = Context(*M, 2.0, 0.4, 2.0, 2.0, *box, precision=precision)
    phi = np.random.default_rng(mx).standard_normal(M[::-1]).astype(dt)
    out = [torch.zeros(M[::-1], dtype=torch.from_numpy(phi).dtype, device="cuda") for _ in range(3)]
    ctx.gauss_efield_on_grid(*box, torch.from_numpy(phi).cuda(), *out)
    for d in range(3):
        inv_h = dt(1.0 / (box[d] / M[d]))
        want = -(np.roll(phi, -1, axis=2 - d) - phi) * inv_h
        assert np.array_equal(out[d].cpu().numpy(), want), d
