"""The eigensolver over matrix sizes at the edges of its reductions (csrc/eig.cu): one row per SM
and the sizes around it, the largest whose rows fit the SMs' shared memory and the next, and the
smallest.

The reduction is backward stable, so an eigenvalue may be off by a modest multiple of
n * eps * ||A||; a vector is held by its residual ||A y - lambda y||, at the bar the kernel tests
hold projectors to.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 9, 64, 151, 152, 153, 305, 1216, 1217])
def test_top_eigenpairs_of_a_hermitian_matrix(n):
    import litho_gb300 as L
    rng = np.random.default_rng(n)
    q = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A = (q + q.conj().T) / 2
    if n == 64:  # a reflector whose column is already zero, and an exactly real row
        A[5, 6:] = 0.0
        A[6:, 5] = 0.0
        A[7] = A[7].real
        A[:, 7] = A[:, 7].real
        A = np.triu(A) + np.triu(A, 1).conj().T
    nk = min(n, 6)
    with L.Context(0) as ctx:
        krn, _, s64 = ctx.calc_kernels(A, nk)
    w = np.linalg.eigvalsh(A)[::-1][:nk]
    norm = np.linalg.norm(A, 2)
    assert np.abs(s64 - w).max() <= 20 * n * np.finfo(float).eps * norm
    y = krn[:, ::-1]
    res = np.linalg.norm(y @ A.T - s64[:, None] * y, axis=1)
    assert res.max() <= 1e-8 * norm
    assert np.abs(y @ y.conj().T - np.eye(nk)).max() <= 1e-8
