"""The order in which calcSOCS adds the bands of its kernel groups (csrc/imaging.cu): one strong kernel
and 31 weak ones, a group each.  The image's mean is the sum of all s_k |K_k M|^2 over the window.  Rounded once
for each weak kernel it would be off by sqrt(31) 0.29 units of 2^-23 (about 1.5e-7, and 1.2e-7 relative where the
sum is 1.3 times a power of two); by three or four it is off by half of that at most.  The strong kernel's own error,
its FFTs', is in the image of that kernel alone too, and is taken out.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_mean_of_the_image():
    import litho_gb300 as L
    nk, N, size = 32, 4, 128
    n, err = (2 * N + 1) ** 2, []
    with L.Context(0) as ctx:
        for seed in range(48):
            rng = np.random.default_rng(seed)
            mr, mi = ctx.fft_mask((rng.random((size, size)) > 0.5).astype(np.float32))
            k = ((rng.standard_normal((nk, n)) + 1j * rng.standard_normal((nk, n))) / 8).astype(np.complex64)
            s = np.where(np.arange(nk) == 0, 1, rng.uniform(0.005, 0.01, nk)).astype(np.float32)
            c = size // 2
            W = (mr + 1j * mi.astype(np.float64))[c - N:c + N + 1, c - N:c + N + 1].reshape(-1)
            power = s.astype(np.float64) * (np.abs(k.astype(np.complex128) * W) ** 2).sum(1)

            def off(scales, want):
                image = ctx.calc_socs(mr, mi, k, scales, N, N, size, size, want_tmpimgp=True)[0]
                return image.astype(np.float64).mean() / want - 1

            err.append(off(s, power.sum()) - off(np.where(np.arange(nk) == 0, s, 0).astype(np.float32), power[0]))
    assert np.sqrt(np.mean(np.square(err))) < 8e-8
