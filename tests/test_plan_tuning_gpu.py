"""Autotuned plans of one process share what tuning found (csrc/batch.cu): a plan whose kernels reach
further in one direction than an earlier plan's gets a conv grid that holds its own intensity band.
Held to the FP64 oracle at the imaging tolerance.
"""
import numpy as np
import pytest

from oracle import np_ref as R

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize("supports", [[(2, 2), (2, 8)], [(10, 10), (10, 16)]])  # (Nx, Ny)
def test_plans_of_equal_nx(supports):
    import litho_gb300 as L
    import torch
    rng = np.random.default_rng(11)
    period, nk, count = 128, 4, 6
    with L.Context(0) as ctx:
        ctx.set_band_method(L.BAND_FFT)
        for nx, ny in supports:
            n = (2 * nx + 1) * (2 * ny + 1)
            k = (rng.standard_normal((nk, n)) + 1j * rng.standard_normal((nk, n))).astype(np.complex64)
            s = rng.uniform(0.1, 1, nk).astype(np.float32)
            masks = (rng.random((count, period, period)) > 0.5).astype(np.float32)
            ks = ctx.kernel_set(k, s, nx, ny)
            plan = L.BatchPlan(ctx, [ks], [period], [(0, period, period)] * count)
            for i, m in enumerate(masks):
                plan.mask(i).copy_(torch.from_numpy(m))
            torch.cuda.synchronize()
            plan.run()
            ctx.synchronize()
            for i, m in enumerate(masks):
                ref = R.mask_to_image(m, k, s, nx, ny)
                assert R.rel_l2(plan.image(i).cpu().numpy(), ref) < TOL, (nx, ny, i, plan.describe())
            plan.close()
            ks.close()
