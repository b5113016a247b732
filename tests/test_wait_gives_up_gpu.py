"""A window whose bounded waits give up (csrc/imaging_fold.cu) leaves NaN in every image, not what happened
to be summed: in the call itself and in those before the flag is read, whose waits end at once.  The
error-path hook makes it happen, as if the rest of the copies had been lost.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,lx,ly,method", [(3, 4, 132, 121, 1), (8, 8, 512, 512, 2), (5, 16, 260, 300, 1), (0, 2, 64, 64, 1)])
@pytest.mark.parametrize("chunk", [0, 1])
def test_images_are_nan(nx, ny, lx, ly, method, chunk):
    import litho_gb300 as L
    import torch
    rng = np.random.default_rng(lx)
    n, batch = (2 * nx + 1) * (2 * ny + 1), 3
    k = (rng.standard_normal((4, n)) + 1j * rng.standard_normal((4, n))).astype(np.complex64)
    with L.Context(0) as ctx:
        ctx.set_band_method(method)
        ks = ctx.kernel_set(k, rng.uniform(0.1, 1, 4).astype(np.float32), nx, ny)
        masks = torch.from_numpy((rng.random((batch, ly, lx)) > 0.5).astype(np.float32)).cuda()
        ragged = torch.from_numpy((rng.random((batch, ly, lx - 1)) > 0.5).astype(np.float32)).cuda()
        torch.cuda.synchronize()
        good = ctx.image_batch(ks, masks, precision=L.PREC_MIXED), ctx.image_batch(ks, ragged)
        ctx.synchronize()
        ctx.set_test_stall(chunk)
        lost = ctx.image_batch(ks, masks, precision=L.PREC_MIXED)
        ctx.set_test_stall(-1)
        after = ctx.image_batch(ks, ragged)
        with pytest.raises(L.LithoError) as ei:
            ctx.synchronize()
        assert ei.value.status == L.LITHO_ERR_TIMEOUT
        assert bool(torch.isnan(lost).all()) and bool(torch.isnan(after).all())
        again = ctx.image_batch(ks, masks, precision=L.PREC_MIXED), ctx.image_batch(ks, ragged)
        ctx.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(good, again))
        ks.close()
