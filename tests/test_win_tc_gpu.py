"""The mixed form's window of large batches above a half-support of 8, or whose masks fill a part of their
period's rows (csrc/imaging_tc.cu): just past the size where it takes over, a width that doesn't fill its 64-column chunks, heights that don't fill its
128-row blocks, rectangular supports, masks exact in TF32 and grey ones; and back-to-back calls.

Held to the FP32 form at the mixed form's bar for a contraction (split TF32: about 2^-22 a product, a
few 1e-6 in relative L2 after the sums).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,ly,lx,nx,ny", [(32, 2048, 2048, 16, 16), (66, 1626, 1268, 12, 13), (84, 1300, 1236, 7, 16),
                                           (512, 512, 512, 10, 9), (110, 600, 1020, 8, 8), (220, 300, 1024, 3, 2)])
@pytest.mark.parametrize("grey", [False, True])
def test_large_batches(B, ly, lx, nx, ny, grey):
    import litho_gb300 as L
    import torch
    assert B * ly * lx >= (2 ** 26 if ny <= 8 else 2 ** 27)
    rng = np.random.default_rng(B)
    n = (2 * nx + 1) * (2 * ny + 1)
    k = (rng.standard_normal((4, n)) + 1j * rng.standard_normal((4, n))).astype(np.complex64)
    s = rng.uniform(0.1, 1, 4).astype(np.float32)
    g = torch.Generator(device="cuda").manual_seed(B)
    masks = torch.rand((B, ly, lx), generator=g, device="cuda")
    if not grey:
        masks = (masks > 0.5).float()
    with L.Context(0) as ctx:
        ks = ctx.kernel_set(k, s, nx, ny)
        plain, mixed, again = (torch.zeros_like(masks) for _ in range(3))
        torch.cuda.synchronize()
        ctx.image_batch(ks, masks, plain)
        ctx.image_batch(ks, masks, mixed, precision=L.PREC_MIXED)
        ctx.image_batch(ks, masks, again, precision=L.PREC_MIXED)
        ctx.synchronize()
        err = (mixed - plain).flatten(1).norm(dim=1) / plain.flatten(1).norm(dim=1)
        assert float(err.max()) < 2e-5
        assert torch.equal(mixed, again)
        ks.close()
