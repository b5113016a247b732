"""The interpolation rows of an early-launched chain read the column twiddles of the image before they wait for
the stage before them (csrc/imaging.cu), so that table is made before the chain's first stage, also in a
plan none of whose masks is as wide as its period (csrc/batch.cu).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec_name,nx,ny", [("fp32", 4, 4), ("mixed", 4, 4), ("mixed", 12, 12)])
def test_tables_come_before_the_window(prec_name, nx, ny):
    import litho_gb300 as L
    import torch
    from torch.profiler import ProfilerActivity, profile
    rng = np.random.default_rng(nx)
    n = (2 * nx + 1) * (2 * ny + 1)
    k = (rng.standard_normal((3, n)) + 1j * rng.standard_normal((3, n))).astype(np.complex64)
    for _ in range(3):  # the profiler's first session of a process may come up after the kernels have run
        with L.Context(0) as ctx:
            ks = ctx.kernel_set(k, rng.uniform(0.1, 1, 3).astype(np.float32), nx, ny)
            ctx.synchronize()
            with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
                plan = L.BatchPlan(ctx, [ks], [256], [(0, 128, 96), (0, 64, 256)],
                                   precision=L.PREC_FP32 if prec_name == "fp32" else L.PREC_MIXED, flags=0)
                ctx.synchronize()
            kernels = sorted((e.time_range.start, e.name) for e in prof.events()
                             if e.device_type == torch.autograd.DeviceType.CUDA)
            plan.close()
            ks.close()
        tables = [t for t, name in kernels if "twF_init" in name]
        if len(tables) == 3:  # widths 128, 64 and 256
            break
    if not kernels:
        pytest.skip("no activity records (another profiler holds them)")
    assert len(tables) == 3 and any("fi_rows" in name for _, name in kernels)
    assert max(tables) < next(t for t, name in kernels if "win_fold" in name or "win_dft" in name)
