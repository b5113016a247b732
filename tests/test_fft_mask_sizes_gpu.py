"""The mask spectrum over row lengths at the edges of its passes (csrc/imaging.cu, fft_rows_centred_kernel):
two to eight points (one pass), every remainder of three stages at a time, rows that don't fill a CTA
and padded ones, up to the longest row; against float64.

A float32 FFT of F points is off by a few eps log2(F) in relative L2: under 5e-6 at any size here.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ly,lx", [(2, 2), (2, 4), (3, 8), (5, 16), (33, 31), (64, 100), (70, 130), (256, 512),
                                   (511, 600), (1025, 1024), (1024, 2048), (3, 4096), (4096, 5), (6, 8192), (8192, 2)])
def test_spectrum(ly, lx):
    import litho_gb300 as L
    rng = np.random.default_rng(ly * 10000 + lx)
    m = rng.standard_normal((ly, lx)).astype(np.float32)
    with L.Context(0) as ctx:
        r, i = ctx.fft_mask(m)
    fy, fx = r.shape
    pad = np.zeros((fy, fx))
    oy, ox = (fy - ly) // 2, (fx - lx) // 2
    pad[oy:oy + ly, ox:ox + lx] = m
    ref = np.fft.fftshift(np.fft.fft2(np.fft.ifftshift(pad))) / (fx * fy)
    got = r.astype(np.float64) + 1j * i.astype(np.float64)
    assert np.linalg.norm(got - ref) <= 5e-6 * np.linalg.norm(ref)
