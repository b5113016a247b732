"""A plan's size classes as branches of its graph (csrc/batch.cu): the images are those of the classes
one after another, bit for bit, over replays back to back; one class, several with different
supports, two that share kernels and period, and one without masks.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLASSES = [(256, 2), (512, 6), (1024, 12), (512, 6), (1024, 3)]  # (period, Nx = Ny)


@pytest.mark.parametrize("used", [(0,), (0, 1), (1, 3), (2, 4), (0, 1, 2, 3, 4)])
@pytest.mark.parametrize("prec_name", ["fp32", "mixed"])
def test_branches_give_the_same_images(used, prec_name):
    import litho_gb300 as L
    import torch
    prec = L.PREC_FP32 if prec_name == "fp32" else L.PREC_MIXED
    rng = np.random.default_rng(7)
    with L.Context(0) as ctx:
        sets = []
        for _, nx in CLASSES:
            k = (rng.standard_normal((5, (2 * nx + 1) ** 2)) + 1j * rng.standard_normal((5, (2 * nx + 1) ** 2)))
            sets.append(ctx.kernel_set(k.astype(np.complex64), rng.uniform(0.1, 1, 5).astype(np.float32), nx, nx))
        periods = [p for p, _ in CLASSES]
        items = [(c, s, s) for c in used for s in (periods[c], periods[c] // 2, periods[c] // 2)]
        masks = [torch.from_numpy((rng.random((y, x)) > 0.5).astype(np.float32)).cuda() for _, x, y in items]
        images = []
        for flags in (0, L.BATCH_GRAPH):
            plan = L.BatchPlan(ctx, sets, periods, items, precision=prec, flags=flags)
            for i, m in enumerate(masks):
                plan.mask(i).copy_(m)
            torch.cuda.synchronize()
            for _ in range(3):
                plan.run()
            ctx.synchronize()
            assert plan.describe()["graph"] is (flags != 0)
            images.append([plan.image(i).clone() for i in range(len(items))])
            plan.close()
        assert all(torch.equal(a, b) for a, b in zip(*images))
        for s in sets:
            s.close()
