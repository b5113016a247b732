"""The FP64 TCC over matrix sizes at the edges of its 32 x 32 tiles and their 16 x 16 quarters, with
so few sources that one share holds them and so many that the last share is partly empty
(csrc/tcc.cu, tcc_fp64_kernel).

The pupil is the same float32 expression on both sides; the bars are those of the oracle comparison
at the usual sizes, and one wrong or missing share is off by at least 1 part in a few hundred.
"""
import numpy as np
import pytest

from oracle import np_ref as R

pytestmark = pytest.mark.gpu


def _period(n, sig):
    """the largest period whose support is n"""
    return max(p for p in range(16, 4096, 16) if R.optics_nx(0.8, p, sig, 193.0) == n)


# n = (2 Nx + 1)(2 Ny + 1): 9, 15, 33, 35, 45, 49, 63, 65, 81, 169
@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 1), (5, 1), (3, 2), (4, 2), (3, 3), (4, 3), (6, 2), (4, 4), (6, 6)])
@pytest.mark.parametrize("size", [5, 21, 101])
def test_tcc_tiles_and_shares(nx, ny, size):
    import litho_gb300 as L
    from litho_gb300 import synth
    src = synth.annular_source(size, 0.5, 0.9)
    sig = R.get_outer_sigma(src)
    Lx, Ly = _period(nx, sig), _period(ny, sig)
    ref = R.calc_tcc(src, sig, 193.0, 0.8, 0.2, Lx, Ly, nx, ny)
    with L.Context(0) as ctx:
        tcc = ctx.calc_tcc(src, sig, 193.0, 0.8, 0.2, Lx, Ly, nx, ny)
    assert np.array_equal(tcc, tcc.conj().T)
    assert np.linalg.norm(tcc - ref) <= 1e-7 * np.linalg.norm(ref)
    assert np.abs(tcc - ref).max() <= 1e-6 * np.abs(ref).max()
