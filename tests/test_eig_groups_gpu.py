"""How the eigensolver shares its work out (csrc/eig.cu): few enough eigenvalues for four SMs each
and one more, a vector's rows over clusters of eight CTAs down to one, blocks of reflectors that
are full, short and single, and rows that end on a chunk of 32 or just past one.

The bars are those of the other sizes: the reduction and the back-transform are backward stable, the
counts are those of a matrix within a few eps ||A||.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nk", [(2, 2), (3, 3), (4, 4), (5, 1), (17, 17), (18, 2), (32, 3), (33, 33), (40, 38),
                                  (40, 39), (64, 19), (65, 25), (97, 76), (97, 77), (160, 153), (289, 24), (321, 50)])
def test_eigenpairs_over_numbers_of_vectors(n, nk):
    import litho_gb300 as L
    rng = np.random.default_rng(1000 * n + nk)
    q = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A = (q + q.conj().T) / 2
    with L.Context(0) as ctx:
        krn, _, s64 = ctx.calc_kernels(A, nk)
    w = np.linalg.eigvalsh(A)[::-1][:nk]
    norm = np.linalg.norm(A, 2)
    assert np.abs(s64 - w).max() <= 20 * n * np.finfo(float).eps * norm
    y = krn[:, ::-1]
    res = np.linalg.norm(y @ A.T - s64[:, None] * y, axis=1)
    assert res.max() <= 1e-8 * norm
    assert np.abs(y @ y.conj().T - np.eye(nk)).max() <= 1e-8
