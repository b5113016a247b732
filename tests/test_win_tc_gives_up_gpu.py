"""The bounded waits of the window on the tensor cores (csrc/imaging_tc.cu), which mixed calls of large sparse
batches take: with the error-path hook its producer is lost before the first chunk, after one, and in
a CTA's second tile.  The kernel leaves, the status is reported, every image is NaN (each has a share in
some CTA that gave up), and later calls repeat the first one's bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grey", [False, True])
def test_producer_lost(grey):
    import litho_gb300 as L
    import torch
    from torch.profiler import ProfilerActivity, profile
    rng = np.random.default_rng(9)
    nx, ny, batch, ly, lx = 5, 3, 220, 300, 1024
    n = (2 * nx + 1) * (2 * ny + 1)
    k = (rng.standard_normal((4, n)) + 1j * rng.standard_normal((4, n))).astype(np.complex64)
    masks = torch.rand((batch, ly, lx), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    if not grey:
        masks = (masks > 0.5).float()
    with L.Context(0) as ctx:
        ks = ctx.kernel_set(k, rng.uniform(0.1, 1, 4).astype(np.float32), nx, ny)
        torch.cuda.synchronize()
        good = ctx.image_batch(ks, masks, precision=L.PREC_MIXED)
        ctx.synchronize()
        names = []
        for _ in range(3):  # the profiler's first session of a process may come up after the kernels have run
            with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
                for chunk in (0, 1, lx // 64 + 3):
                    ctx.set_test_stall(chunk)
                    lost = ctx.image_batch(ks, masks, precision=L.PREC_MIXED)
                    with pytest.raises(L.LithoError) as ei:
                        ctx.synchronize()
                    assert ei.value.status == L.LITHO_ERR_TIMEOUT
                    assert bool(torch.isnan(lost).all())
            names = [e.name for e in prof.events() if "win_" in e.name]
            if names:
                break
        if [e for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]:  # there are activity records
            assert names and all("win_dft_tc" in name for name in names)
        ctx.set_test_stall(-1)
        again = ctx.image_batch(ks, masks, precision=L.PREC_MIXED)
        ctx.synchronize()
        assert torch.equal(good, again)
        ks.close()
