"""The surrogate's column kernel over its group sizes (csrc/fno.cu): one, two and four masks a CTA,
whole groups and a last one that is short, at every grid size, forward and backward.

The group decides who computes a mask, not how: an image doesn't depend on its batch, bit for bit.
Gradients are held to the float64 oracle at the bar for its BF16 operands, a gradient group at a time;
a mask left out or taken twice of at most 57 is off by at least that much in the loss's share.
"""
import numpy as np
import pytest

from oracle import fno_ref as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [64, 128, 256])
@pytest.mark.parametrize("B", [1, 3, 29, 30, 57, 63, 64])
def test_images_do_not_depend_on_the_group(L, B):
    import litho_gb300
    import torch
    from litho_gb300 import surrogate as S
    with litho_gb300.Context(0) as ctx:
        model = S.Surrogate(ctx, L=L, seed=3)
        masks = S.rect_masks(ctx, 5, 0, B, L, wmin=4, wmax=L // 4)
        out = model.forward(masks)
        for b in {0, B // 2, B - 1}:
            assert torch.equal(model.forward(masks[b:b + 1].contiguous())[0], out[b])
        model.close()


@pytest.mark.parametrize("B", [3, 29, 30, 57])
def test_gradients_of_every_group_size(B):
    import litho_gb300
    import torch
    from litho_gb300 import surrogate as S
    L = 64
    with litho_gb300.Context(0) as ctx:
        model = S.Surrogate(ctx, L=L, seed=4)
        masks = S.rect_masks(ctx, 6, 0, B, L, wmin=4, wmax=16)
        m = masks.cpu().numpy()
        tgt = (0.2 + 0.5 * m).astype(np.float32)
        loss, g = model.loss_grad(masks, torch.tensor(tgt, device=masks.device))
        rl, rg = F.loss_and_grad(model.params().astype(np.float64), m, tgt)
        assert abs(loss - rl) <= 2e-2 * rl
        gu, ru = F.unpack(g.astype(np.float64)), F.unpack(rg)
        for name, _ in F.param_shapes():
            assert np.linalg.norm(gu[name] - ru[name]) <= 2e-2 * max(np.linalg.norm(ru[name]), 1e-30), name
        model.close()
