"""Calls of one image or two, whose stages start while the stage before them runs (csrc/imaging.cu): many
calls back to back with different masks, on the same workspaces and without a wait in between, give
each mask its own image, bit for bit what the call gives by itself and the oracle's at float32.
"""
import numpy as np
import pytest

from oracle import np_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ly,lx,nx", [(64, 64, 1), (256, 256, 2), (130, 200, 3), (512, 512, 4), (1024, 1024, 8)])
@pytest.mark.parametrize("B", [1, 2])
def test_back_to_back_calls(ly, lx, nx, B):
    import litho_gb300 as L
    import torch
    rng = np.random.default_rng(ly + lx + B)
    k = (rng.standard_normal((9, (2 * nx + 1) ** 2)) + 1j * rng.standard_normal((9, (2 * nx + 1) ** 2)))
    k, s = k.astype(np.complex64), rng.uniform(0.1, 1, 9).astype(np.float32)
    masks = [torch.from_numpy((rng.random((B, ly, lx)) > 0.5).astype(np.float32)).cuda() for _ in range(6)]
    with L.Context(0) as ctx:
        ks = ctx.kernel_set(k, s, nx, nx)
        alone = []
        for m in masks:
            out = torch.zeros_like(m)
            torch.cuda.synchronize()
            ctx.image_batch(ks, m, out)
            ctx.synchronize()
            alone.append(out)
        outs = [torch.zeros_like(masks[0]) for _ in range(60)]
        torch.cuda.synchronize()
        for i, o in enumerate(outs):
            ctx.image_batch(ks, masks[i % 6], o)
        ctx.synchronize()
        assert all(torch.equal(o, alone[i % 6]) for i, o in enumerate(outs))
        ks.close()
    if min(lx, ly) >= 128:  # (the oracle interpolates upwards from its 128 x 128 grid)
        ref = R.mask_to_image(masks[0][0].cpu().numpy(), k, s, nx, nx, 128, None)
        assert R.rel_l2(alone[0][0].cpu().numpy(), ref) < 1e-5
