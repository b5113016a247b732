"""Several contexts solving at once, each on its own thread and stream: the reduction's one launch per
matrix (csrc/eig.cu) shares the SMs with the others', small and as large as its rows fit.  Every
thread gets what the calls give one at a time, bit for bit.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(289, 289, 289), (1089, 1089), (1216, 65, 1089)])
def test_solves_at_once(sizes):
    import litho_gb300 as L
    rng = np.random.default_rng(sum(sizes))
    mats = []
    for n in sizes:
        q = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        mats.append((q + q.conj().T) / 2)
    alone = []
    for A in mats:
        with L.Context(0) as ctx:
            alone.append(ctx.calc_kernels(A, 8))
    got, errors = [None] * len(mats), []

    def solve(i):
        try:
            with L.Context(0) as ctx:
                got[i] = [ctx.calc_kernels(mats[i], 8) for _ in range(4)]
        except Exception as e:  # reported below, by the thread that asserts
            errors.append(e)

    threads = [threading.Thread(target=solve, args=(i,)) for i in range(len(mats))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for ref, runs in zip(alone, got):
        for run in runs:
            assert all(np.array_equal(a, b) for a, b in zip(ref, run))
