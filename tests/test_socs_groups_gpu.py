"""calcSOCS with its intensity wanted, over numbers of kernels: one group, one kernel a group up to the
most groups, and several kernels a group with a short last one (litho_calc_socs); every convolution
grid, and a period whose spectrum is larger than the image.

Held to the oracle at the bar of the other SOCS images (float32 transforms).
"""
import numpy as np
import pytest

from oracle import np_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conv_n,embed", [(128, 94), (64, None), (32, None)])
@pytest.mark.parametrize("nk", [1, 2, 31, 32, 33, 70])
def test_intensity_over_numbers_of_kernels(conv_n, embed, nk):
    import litho_gb300 as L
    rng = np.random.default_rng(nk)
    nx, ny, lx, ly = 3, 4, 200, 128
    krns = rng.standard_normal((nk, 2 * ny + 1, 2 * nx + 1)) + 1j * rng.standard_normal((nk, 2 * ny + 1, 2 * nx + 1))
    krns = krns.reshape(nk, -1).astype(np.complex64)
    scales = rng.uniform(0.1, 1.0, nk).astype(np.float32)
    mskf = R.ft_r2c_padded((rng.random((ly, lx)) > 0.5).astype(np.float32), 256, 128)
    ref_img, ref_tmp = R.calc_socs(mskf, lx, ly, krns, scales, nk, nx, ny, conv_n, embed)
    with L.Context(0) as ctx:
        img, tmp = ctx.calc_socs(mskf.real.astype(np.float32), mskf.imag.astype(np.float32), krns, scales, nx, ny, lx, ly,
                                 want_tmpimgp=True, conv_n=conv_n)
    assert R.rel_l2(tmp, ref_tmp) < 1e-5
    assert R.rel_l2(img, ref_img) < 1e-5
