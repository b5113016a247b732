"""Several contexts calling at once, each on its own thread and stream, with sizes that ask for different
amounts of shared memory from the same kernels: every thread gets what its calls give alone, bit for
bit, and no call is refused.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kernels(rng, nx, ny, nk):
    n = (2 * nx + 1) * (2 * ny + 1)
    k = (rng.standard_normal((nk, n)) + 1j * rng.standard_normal((nk, n))).astype(np.complex64)
    return k, rng.uniform(0.1, 1, nk).astype(np.float32)


def _imager(nx, ny, B, ly, lx, prec, method):
    def make(ctx):
        import litho_gb300 as L
        import torch
        rng = np.random.default_rng(B + lx)
        ctx.set_band_method(method)
        ks = ctx.kernel_set(*_kernels(rng, nx, ny, 6), nx, ny)
        gen = torch.Generator(device="cuda").manual_seed(B + lx)
        masks = (torch.rand((B, ly, lx), generator=gen, device="cuda") > 0.5).float()
        out = torch.zeros_like(masks)
        torch.cuda.synchronize()
        return lambda: ctx.image_batch(ks, masks, out, precision=prec), lambda: out.cpu().numpy()
    return make


def _spectrum(side):
    def make(ctx):
        mask = np.random.default_rng(side).random((side, side)).astype(np.float32)
        got = []
        return lambda: got.__setitem__(slice(None), ctx.fft_mask(mask)), lambda: np.stack(got)
    return make


def _surrogate(side, B):
    def make(ctx):
        from litho_gb300 import surrogate as S
        model = S.Surrogate(ctx, L=side, seed=3)
        masks = S.rect_masks(ctx, 5, 0, B, side, wmin=4, wmax=16)
        ctx.synchronize()
        got = []
        return lambda: got.__setitem__(slice(None), [model.loss_grad(masks, masks)[1]]), lambda: np.stack(got)
    return make


def _sets():
    import litho_gb300 as L
    return {
        # one support, batches whose window, band, rows and image kernels all ask for different sizes
        "batches": (400, [_imager(8, 8, B, 1024, 1024, L.PREC_FP32, L.BAND_AUTO) for B in (1, 16, 64, 256)]),
        "supports": (400, [_imager(8, ny, B, 512, 500, L.PREC_MIXED, m) for ny, B, m in
                           ((8, 2, L.BAND_TCC), (3, 40, L.BAND_TCC), (7, 9, L.BAND_FFT), (5, 1, L.BAND_FFT))]),
        "large": (200, [_imager(nx, 16, B, 1024, 1024, L.PREC_MIXED, L.BAND_FFT) for nx, B in ((16, 1), (12, 20), (16, 8))]),
        "ragged": (400, [_imager(6, 6, B, 303, 411, L.PREC_FP32, L.BAND_FFT) for B in (1, 30, 200)]),
        "spectra": (60, [_spectrum(s) for s in (60, 500, 1000, 2000)]),
        "surrogates": (60, [_surrogate(64, 3), _surrogate(128, 2), _surrogate(256, 1)]),
    }


@pytest.mark.parametrize("name", ["batches", "supports", "large", "ragged", "spectra", "surrogates"])
def test_calls_at_once(name):
    import litho_gb300 as L
    rounds, makers = _sets()[name]
    alone = []
    for make in makers:
        with L.Context(0) as ctx:
            call, result = make(ctx)
            call()
            ctx.synchronize()
            alone.append(result())
    got, errors, gate = [None] * len(makers), [], threading.Barrier(len(makers))

    def work(i):
        try:
            with L.Context(0) as ctx:
                call, result = makers[i](ctx)
                call()
                gate.wait()
                for _ in range(rounds):
                    call()
                ctx.synchronize()
                got[i] = result()
        except Exception as e:  # reported below, by the thread that asserts
            errors.append((i, e))
            gate.abort()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(makers))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert all(np.array_equal(a, b) for a, b in zip(alone, got))
