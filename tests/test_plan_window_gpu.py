"""Mixed plans whose classes ask the tensor cores for the window first (csrc/batch.cu, plan_win_tc): several mask
sizes to a launch, more sizes than one launch takes, heights that don't fill 128-row blocks, widths that
don't fill 64-column chunks; above a half-support of 8 and, with masks that fill half of their period or
less, below.

Binary masks are held to the plain form at the bar of a split-TF32 contraction (about 2^-22 a product).
Grey masks are left to the folded kernel: up to a half-support of 8, where everything else is the plain
form's too, their images are the plain plan's bit for bit.  A batch that changes from one kind to the
other between runs of a graph, and one grey mask that the samples may miss.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [  # period, Nx, Ny, (count, rows, columns) per size
    (1024, 12, 9, [(40, 1024, 1024), (30, 900, 1000), (5, 130, 68)]),
    (2048, 16, 16, [(8, 2048, 2048), (7, 1502, 2044), (6, 1998, 1240), (3, 2, 4), (9, 1030, 1024), (2, 128, 64)]),
    (1024, 8, 8, [(100, 512, 512), (20, 300, 260)]),
    (512, 4, 3, [(310, 256, 256), (90, 130, 388), (2, 512, 512)]),
]


def _images(L, ctx, ks, period, items, masks, prec, flags, kinds):
    import torch
    plan = L.BatchPlan(ctx, [ks], [period], items, precision=prec, flags=flags)
    out = []
    for kind in kinds:
        for i, m in enumerate(masks[kind]):
            plan.mask(i).copy_(m)
        torch.cuda.synchronize()
        plan.run()
        plan.run()
        ctx.synchronize()
        out.append(torch.stack([plan.image(i) for i in range(len(items))]))
    plan.close()
    return out


@pytest.mark.parametrize("period,nx,ny,sizes", CASES)
@pytest.mark.parametrize("graph", [False, True])
def test_plan_windows(period, nx, ny, sizes, graph):
    import litho_gb300 as L
    import torch
    rng = np.random.default_rng(nx)
    n = (2 * nx + 1) * (2 * ny + 1)
    k = (rng.standard_normal((3, n)) + 1j * rng.standard_normal((3, n))).astype(np.complex64)
    assert sum(c * y * x for c, y, x in sizes) >= (1 << 26 if ny > 8 else 3 << 23)
    assert ny > 8 or 2 * sum(c * y for c, y, _ in sizes) <= period * sum(c for c, _, _ in sizes)
    items = [(0, x, y) for c, y, x in sizes for _ in range(c)]
    gen = torch.Generator(device="cuda").manual_seed(ny)
    grey = [torch.rand((y, x), generator=gen, device="cuda") for _, x, y in items]
    binary = [(m > 0.5).float() for m in grey]
    masks = dict(grey=grey, binary=binary, one=binary[:1] + grey[1:2] + binary[2:])
    kinds = ["binary", "grey", "binary", "one"]
    with L.Context(0) as ctx:
        ks = ctx.kernel_set(k, rng.uniform(0.1, 1, 3).astype(np.float32), nx, ny)
        plain = _images(L, ctx, ks, period, items, masks, L.PREC_FP32, 0, ["binary", "grey", "one"])
        plain = [plain[0], plain[1], plain[0], plain[2]]
        mixed = _images(L, ctx, ks, period, items, masks, L.PREC_MIXED, L.BATCH_GRAPH if graph else 0, kinds)
        for a, b in zip(plain, mixed):
            assert float(((a - b).flatten(1).norm(dim=1) / a.flatten(1).norm(dim=1)).max()) < 2e-5
        assert torch.equal(mixed[0], mixed[2])
        if ny <= 8:
            assert torch.equal(mixed[1], plain[1])
            assert not torch.equal(mixed[0], plain[0])  # the tensor cores did them
        ks.close()
