"""Performance cases of the aerial-image framework: what a user's program calls, over the sizes it calls it with.

Three programs stand behind them.  A mask-imaging service keeps one kernel set per optical configuration and images
batches of device tensors (both precisions, binary layouts and 8-bit grey masks, one mask or a thousand, ragged
sizes), batches that arrive in host memory, and mixed sizes through a batch plan.  An optics program goes from a
source to its TCC, its kernels and a first image, or calls the reference program's own functions one by one
(FT_r2c_padded, calcSOCS) on host arrays.  A surrogate program trains the network and images with it.

``exact`` restates each in 64 bits with numpy and torch alone.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fpga-litho-accel_gb300"))

NA, WAVELENGTH, SIGMA = 0.8, 193.0, 0.9
DEV = "cuda"


# --------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one small clip, as an interactive tool or a correction loop images it: launches and latency
        dict(name="image_one_256", kind="image", B=1, Ly=256, Lx=256, nk=24, prec="fp32", grey=False),
        # the plain form on a batch of full-size layouts
        dict(name="image_fp32_1024", kind="image", B=256, Ly=1024, Lx=1024, nk=24, prec="fp32", grey=False),
        # clips cut to their content: odd sides, rows that start at no particular alignment
        dict(name="image_fp32_ragged", kind="image", B=40, Ly=913, Lx=777, nk=24, prec="fp32", grey=True),
        # the benchmark's step: 1024 layouts, mixed precision
        dict(name="image_mixed_1024", kind="image", B=1024, Ly=1024, Lx=1024, nk=24, prec="mixed", grey=False),
        # grey-level masks (the reference's PNG masks are), whose values have no short form
        dict(name="image_mixed_grey_1024", kind="image", B=256, Ly=1024, Lx=1024, nk=24, prec="mixed", grey=True),
        # sixty masks of five sizes in two size classes, one graph launch
        dict(name="plan_uneven_60", kind="plan", counts="256:12,512:12,768:12,1024:14,2048:10", nk=24, prec="mixed"),
        # masks that arrive in pinned host memory and images that go back there
        dict(name="image_host_1024", kind="host", B=64, Ly=1024, Lx=1024, nk=24, prec="mixed", grey=False),
        # the reference program's own calls on host arrays: mask spectrum, then calcSOCS with its conv-grid image
        dict(name="reference_calls_1024", kind="calls", Ly=1024, Lx=1024, nk=10),
        # a new optical configuration at 1024 (TCC 289 x 289): source to first image, FP64 throughout
        dict(name="optics_1024", kind="optics", L=1024, nk=24, points=2000, tcc="fp64"),
        # the same at 2048 (TCC 1089 x 1089) with the tensor-core TCC
        dict(name="optics_2048", kind="optics", L=2048, nk=24, points=2000, tcc="split"),
        # surrogate inference with its error estimate
        dict(name="surrogate_predict_256", kind="predict", B=64, L=256),
        # surrogate training: loss and all gradients of one mini-batch
        dict(name="surrogate_grad_256", kind="grad", B=32, L=256),
    ]


def draw(rng):
    kind = rng.choice(["image"] * 6 + ["plan", "host", "calls", "optics", "predict", "grad"])
    nk = rng.choice([8, 16, 24, 24, 32])

    def side(step=1):
        return max(step, int(round(128 * 2 ** (4 * rng.random()) / step)) * step)

    if kind in ("image", "host"):
        prec = rng.choice(["fp32", "mixed"])
        Lx, Ly = side(4 if prec == "mixed" else 1), side()
        most = max(1, min(1024, (1 << (27 if kind == "host" else 29)) // (Lx * Ly)))
        B = max(1, int(round(math.exp(rng.random() * math.log(most)))))
        return dict(kind=kind, B=B, Ly=Ly, Lx=Lx, nk=nk, prec=prec, grey=rng.random() < 0.4)
    if kind == "plan":
        sizes = rng.sample([256, 384, 512, 640, 768, 896, 1024, 2048], 4)
        return dict(kind=kind, counts=",".join("%d:%d" % (s, rng.randint(2, 14)) for s in sorted(sizes)), nk=nk,
                    prec=rng.choice(["fp32", "mixed"]))
    if kind == "calls":
        return dict(kind=kind, Ly=side(), Lx=side(), nk=rng.choice([6, 10, 20, 24]))
    if kind == "optics":
        return dict(kind=kind, L=rng.choice([512, 768, 1024, 1280, 1536]), nk=nk, points=rng.randint(300, 2500),
                    tcc=rng.choice(["fp64", "fp64", "split"]))
    return dict(kind=kind, B=rng.randint(4, 96 if kind == "predict" else 48), L=rng.choice([128, 256]))


# ------------------------------------------------------------------------------------------ optics (numpy, FP64)
def pow2(n):
    return 1 << max(0, (n - 1).bit_length())


def half_support(L):
    """floor(NA L (1 + sigma) / lambda), at least 1."""
    return max(1, int(math.floor(np.float32(NA) * np.float32(L) * np.float32(1 + SIGMA) / np.float32(WAVELENGTH))))


def quasar(S, weights=None):
    """Four poles on the diagonals, sigma 0.7 to 0.9, 30 degrees wide, on an S x S grid; `weights`: their pixels' intensities."""
    c = (S - 1) // 2
    y, x = np.mgrid[0:S, 0:S].astype(np.float64) - c
    r = np.hypot(x, y) / c
    a = np.degrees(np.arctan2(y, x)) % 90.0
    lit = (r >= 0.7) & (r <= SIGMA) & (np.abs(a - 45.0) <= 15.0)
    src = lit.astype(np.float64) if weights is None else lit * weights
    return (src / src.sum()).astype(np.float32)


def pupil(src, Lx, Ly, Nx, Ny, defocus):
    """(P, J): the pupil of every lit source point on the window (rows of 2Nx+1), its coordinates rounded as 32-bit
    programs round them (they decide which points are inside), the phase in 64 bits."""
    f = np.float32
    sh = (src.shape[0] - 1) // 2
    q, p = np.nonzero(src)
    J = src[q, p].astype(np.float64)
    sx, sy = ((p - sh).astype(f) / f(sh))[None], ((q - sh).astype(f) / f(sh))[None]
    lx, ly = f(f(Lx) * f(NA)) / f(WAVELENGTH), f(f(Ly) * f(NA)) / f(WAVELENGTH)
    ny, nx = (v.reshape(-1, 1) for v in np.mgrid[-Ny:Ny + 1, -Nx:Nx + 1])
    fy, fx = ny.astype(f) / ly + sy, nx.astype(f) / lx + sx
    rho2 = (fx * fx + fy * fy).astype(f)
    inside = (fy * fy <= 1) & (rho2 <= 1)
    dz = f(defocus) / f(f(f(NA) * f(NA)) / f(WAVELENGTH))
    dzk = f(dz * f(2 * math.pi / WAVELENGTH))
    r = (rho2 * f(NA) * f(NA)).astype(np.float64)
    return inside * np.exp(1j * float(dzk) * np.sqrt(np.maximum(0.0, 1.0 - r))), J


def top_kernels(P, J, nk):
    """(kernels [nk][n], scales [nk]): the largest eigenpairs of P diag(J) P^H, each eigenvector reversed."""
    A = P * np.sqrt(J)
    w, v = np.linalg.eigh(A @ A.conj().T)
    return np.ascontiguousarray(v[:, ::-1][:, :nk].T[:, ::-1]), w[::-1][:nk].copy()


@functools.lru_cache(maxsize=None)
def kernels(Fx, Fy, nk):
    """The kernel set a program keeps for its optics: period Fx x Fy, quasar source, in focus."""
    Nx, Ny = half_support(Fx), half_support(Fy)
    nk = min(nk, (2 * Nx + 1) * (2 * Ny + 1))
    K, s = top_kernels(*pupil(quasar(61), Fx, Fy, Nx, Ny, 0.0), nk)
    return K.reshape(nk, 2 * Ny + 1, 2 * Nx + 1), s.astype(np.float32), Nx, Ny


# ------------------------------------------------------------------------------------------------------- masks
def layouts(seed, B, Ly, Lx, grey=False):
    """B layouts on the GPU: rectangles and lines of 8 to 96 pixels, about 40 % covered; `grey`: 8-bit levels over 255."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + B * 31 + Ly * 17 + Lx)
    out = torch.empty(B, Ly, Lx, device=DEV)
    R = max(6, min(96, Ly * Lx // 6000))
    x, y = torch.arange(Lx, device=DEV), torch.arange(Ly, device=DEV)
    for b in range(0, B, 64):
        n = min(64, B - b)

        def spans(size, at):
            w = torch.randint(8, max(9, min(97, size // 2)), (n, R, 1), generator=g, device=DEV)
            o = (torch.rand(n, R, 1, generator=g, device=DEV) * (size - w)).long()
            return ((at >= o) & (at < o + w)).half()

        rows, cols = spans(Ly, y), spans(Lx, x)
        m = (rows.transpose(1, 2) @ cols > 0.5).float()
        if grey:
            m = (m * 200 + torch.randint(0, 56, m.shape, generator=g, device=DEV)) / 255.0
        out[b:b + n] = m
    return out


def context():
    import litho_gb300 as L
    return L, L.Context(0)


def on_torch_stream(ctx):
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)


def prec_of(L, case):
    return L.PREC_MIXED if case["prec"] == "mixed" else L.PREC_FP32


def sizes_of(case):
    return [(int(s), int(n)) for s, n in (t.split(":") for t in case["counts"].split(","))]


def points_grid(points):
    """The odd source grid whose quasar has about `points` lit pixels."""
    return max(21, 2 * int(round(math.sqrt(points / (math.pi * (0.81 - 0.49) / 3.0)))) + 1)


# ----------------------------------------------------------------------------------------------- network weights
C, M, H, NL = 32, 16, 128, 4


def weights(seed):
    """The network's parameters in the library's flat order (Pw, Pb, W, Wb, R, Q1, q1b, Q2, q2b)."""
    r = np.random.default_rng(seed)
    parts = [r.normal(0, 1, C), r.normal(0, 0.1, C), r.normal(0, 1 / math.sqrt(C), NL * C * C), r.normal(0, 0.05, NL * C),
             r.random(NL * 2 * M * M * C * C * 2, dtype=np.float32) / (C * C),
             r.normal(0, 1 / math.sqrt(C), H * C), r.normal(0, 0.05, H), r.normal(0, 1 / math.sqrt(H), H), r.normal(0, 0.05, 1)]
    return np.concatenate([np.asarray(p, np.float32).ravel() for p in parts])


def network(theta, masks):
    """The FNO-2d in the type of its inputs: lift, four Fourier layers, projection."""
    at = [0]

    def take(*shape):
        n = int(np.prod(shape))
        at[0] += n
        return theta[at[0] - n:at[0]].reshape(shape)

    Pw, Pb, W, Wb = take(C), take(C), take(NL, C, C), take(NL, C)
    R, Q1, q1b, Q2, q2b = take(NL, 2 * M, M, C, C, 2), take(H, C), take(H), take(H), take(1)
    B, L, _ = masks.shape
    v = masks[..., None] * Pw + Pb
    ky = torch.cat([torch.arange(M), torch.arange(L - M, L)]).to(masks.device)
    for l in range(NL):
        low = torch.fft.rfft2(v, dim=(1, 2))[:, ky, :M, :]
        mixed = torch.einsum("bjkc,jkco->bjko", low, torch.view_as_complex(R[l].contiguous()))
        full = torch.zeros(B, L, L // 2 + 1, C, dtype=mixed.dtype, device=masks.device)
        full[:, ky, :M, :] = mixed
        z = v @ W[l].T + Wb[l] + torch.fft.irfft2(full, s=(L, L), dim=(1, 2))
        v = torch.nn.functional.gelu(z, approximate="tanh") if l < NL - 1 else z
    return torch.nn.functional.gelu(v @ Q1.T + q1b, approximate="tanh") @ Q2 + q2b[0]


# ------------------------------------------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("image", "host"):
        L, ctx = context()
        K, s, Nx, Ny = kernels(pow2(case["Lx"]), pow2(case["Ly"]), case["nk"])
        ks = ctx.kernel_set(K, s, Nx, Ny)
        masks = layouts(seed, case["B"], case["Ly"], case["Lx"], case["grey"])
        st = dict(kind=kind, ctx=ctx, ks=ks, prec=prec_of(L, case))
        if kind == "host":  # pinned buffers the program keeps for its transfers
            st["masks"] = masks.cpu().pin_memory().numpy()
            st["images"] = torch.empty(masks.shape, pin_memory=True).numpy()
        else:
            on_torch_stream(ctx)
            st["masks"], st["images"] = masks, torch.empty_like(masks)
        return st
    if kind == "plan":
        L, ctx = context()
        items, sets = [], []
        periods = sorted({1024 if s <= 1024 else 2048 for s, _ in sizes_of(case)})
        for p in periods:
            K, s, Nx, Ny = kernels(p, p, case["nk"])
            sets.append(ctx.kernel_set(K, s, Nx, Ny))
        for s, n in sizes_of(case):
            items += [(periods.index(1024 if s <= 1024 else 2048), s, s)] * n
        plan = L.BatchPlan(ctx, sets, periods, items, prec_of(L, case))
        on_torch_stream(ctx)
        at = 0
        for s, n in sizes_of(case):
            for m in layouts(seed, n, s, s):
                plan.mask(at).copy_(m)
                at += 1
        images = [plan.image(i) for i in range(len(items))]
        for t in images:  # views of the plan's memory: who keeps one keeps the plan
            t.owner = (plan, sets, ctx)
        return dict(kind=kind, ctx=ctx, sets=sets, plan=plan, images=images)
    if kind == "calls":
        L, ctx = context()
        K, s, Nx, Ny = kernels(pow2(case["Lx"]), pow2(case["Ly"]), case["nk"])
        return dict(kind=kind, ctx=ctx, mask=layouts(seed, 1, case["Ly"], case["Lx"], True)[0].cpu().numpy(), K=K, s=s,
                    Nx=Nx, Ny=Ny)
    if kind == "optics":
        L, ctx = context()
        on_torch_stream(ctx)
        src, N, defocus = optics_of(case, seed)
        if case["tcc"] == "split":
            ctx.tcc_gemm_shape(128, 64, 0)  # results that repeat bit for bit
        masks = layouts(seed, 1, case["L"], case["L"])
        return dict(kind=kind, ctx=ctx, src=src, N=N, defocus=defocus, L=case["L"], nk=case["nk"], masks=masks,
                    images=torch.empty_like(masks), split=case["tcc"] == "split")
    from litho_gb300 import surrogate as S
    L, ctx = context()
    net = S.Surrogate(ctx, case["L"], seed=1)
    net.set_params(weights(seed))
    masks = layouts(seed, case["B"], case["L"], case["L"])
    st = dict(kind=kind, ctx=ctx, net=net, masks=masks)
    K, s, Nx, Ny = kernels(case["L"], case["L"], 24)
    ks = ctx.kernel_set(K, s, Nx, Ny)
    if kind == "predict":
        return dict(st, ks=ks, images=torch.empty_like(masks))
    return dict(st, targets=aerial(masks, K, s, Nx, Ny).float())


def optics_of(case, seed):
    """A freeform quasar source (pixel intensities from the seed), its window and a defocus."""
    r = np.random.default_rng(seed)
    S = points_grid(case["points"])
    src = quasar(S, r.uniform(0.5, 1.0, (S, S)))
    return src, half_support(case["L"]), float(np.float32(r.uniform(-0.3, 0.3)))


# ---------------------------------------------------------------------------------------------------------- run
def run(st):
    kind, ctx = st["kind"], st["ctx"]
    if kind in ("image", "host"):
        return ctx.image_batch(st["ks"], st["masks"], st["images"], precision=st["prec"])
    if kind == "plan":
        st["plan"].run()
        return st["images"]
    if kind == "calls":
        fr, fi = ctx.fft_mask(st["mask"])
        Ly, Lx = st["mask"].shape
        image, conv = ctx.calc_socs(fr, fi, st["K"], st["s"], st["Nx"], st["Ny"], Lx, Ly, want_tmpimgp=True)
        return [fr, fi, image, conv]
    if kind == "optics":
        import litho_gb300 as L
        N, Lp = st["N"], st["L"]
        tcc = ctx.calc_tcc(st["src"], SIGMA, WAVELENGTH, NA, st["defocus"], Lp, Lp, N, N,
                           precision=L.TCC_SPLIT_BF16 if st["split"] else L.TCC_FP64)
        K, s32, s64 = ctx.calc_kernels(tcc, st["nk"])
        ks = ctx.kernel_set(K, s32, N, N)
        ctx.image_batch(ks, st["masks"], st["images"])
        torch.cuda.current_stream().synchronize()  # the program looks at its first image
        ks.close()
        return [tcc, s32, s64, st["images"]]
    if kind == "predict":
        return list(st["net"].predict(st["ks"], st["masks"], st["images"]))
    loss, grad = st["net"].loss_grad(st["masks"], st["targets"])
    return [loss, grad]


# --------------------------------------------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]

    def imaging(B, my, mx, Ly, Lx, N, M_):
        # mask in, image out; the two pruned transforms at the cost of their contractions with the four-fold symmetry
        # of cos and sin used, as FFT programs use it
        return 4.0 * B * (my * mx + Ly * Lx), B * (my * mx * (2 * N + 1) / 2.0 + Ly * Lx * (4 * M_ + 1) / 2.0)

    if kind in ("image", "host", "calls"):
        B, Ly, Lx = case.get("B", 1), case["Ly"], case["Lx"]
        Nx, Ny = half_support(pow2(Lx)), half_support(pow2(Ly))
        b, f = imaging(B, Ly, Lx, Ly, Lx, Nx, Ny)
        if kind == "calls":  # the whole spectrum is an output of the first call
            F = pow2(Lx) * pow2(Ly)
            b, f = b + 8.0 * F, f + 2.5 * F * math.log2(F)
        return dict(bytes=b + 8.0 * case["nk"] * (2 * Nx + 1) * (2 * Ny + 1), flops=f)
    if kind == "plan":
        b = f = 0.0
        for s, n in sizes_of(case):
            p = 1024 if s <= 1024 else 2048
            x, y = imaging(n, s, s, p, p, half_support(p), half_support(p))
            b, f = b + x, f + y
        return dict(bytes=b, flops=f)
    if kind == "optics":
        n = (2 * half_support(case["L"]) + 1) ** 2
        # TCC to the host and back; Hermitian contraction and tridiagonalisation
        return dict(bytes=32.0 * n * n + 8.0 * case["L"] ** 2, flops=4.0 * case["points"] * n * n + 16.0 / 3 * n ** 3)
    px = float(case["B"] * case["L"] ** 2)
    layer = 2.0 * C * C + 2 * 4.0 * M * C  # per pixel: W v and the two row transforms
    f = px * (NL * layer + 2.0 * C * H)
    act = px * C * 2  # one layer's activations, 16 bits
    if kind == "predict":
        return dict(bytes=act * 2 * (NL - 1) + 8 * px + 4.0 * weights_count(), flops=f)
    return dict(bytes=act * 4 * NL + 8 * px + 8.0 * weights_count(), flops=3 * f)


def weights_count():
    return 2 * C + NL * C * C + NL * C + NL * 2 * M * M * C * C * 2 + H * C + 2 * H + 1


# -------------------------------------------------------------------------------------------------------- exact
def aerial(masks, K, s, Nx, Ny, Fx=None, Fy=None, crop=True, conv=None):
    """SOCS images of `masks` in 64 bits by whole FFTs: centred in a period Fx x Fy, spectrum, K fields on a grid,
    intensity, interpolation to the period, cropped to the masks' size. `conv`: also the intensity on that grid."""
    B, h, w = masks.shape
    Fx, Fy = Fx or pow2(w), Fy or pow2(h)
    n = conv or max(32, pow2(4 * max(Nx, Ny) + 1))
    Kt = torch.as_tensor(np.asarray(K)).to(DEV).to(torch.complex64).to(torch.complex128).reshape(-1, 2 * Ny + 1, 2 * Nx + 1)
    st = torch.as_tensor(np.asarray(s, np.float32)).to(DEV).double()
    vy, vx = torch.arange(-Ny, Ny + 1, device=DEV), torch.arange(-Nx, Nx + 1, device=DEV)
    oy, ox = (Fy - h) // 2, (Fx - w) // 2
    by, bx = torch.arange(-2 * Ny, 2 * Ny + 1, device=DEV), torch.arange(-2 * Nx, 2 * Nx + 1, device=DEV)
    out = torch.empty((B, h, w) if crop else (B, Fy, Fx), dtype=torch.float64, device=DEV)
    step = max(1, (1 << 25) // (Fx * Fy))
    grid = spec = None
    for b in range(0, B, step):
        m = masks[b:b + step]
        pad = torch.zeros(m.shape[0], Fy, Fx, dtype=torch.float64, device=DEV)
        pad[:, oy:oy + h, ox:ox + w] = m.double()
        spec = torch.fft.fft2(torch.fft.ifftshift(pad, dim=(1, 2))) / (Fx * Fy)
        W = spec[:, vy % Fy][:, :, vx % Fx]
        inten = torch.zeros(m.shape[0], n, n, dtype=torch.float64, device=DEV)
        for k in range(Kt.shape[0]):
            E = torch.zeros(m.shape[0], n, n, dtype=torch.complex128, device=DEV)
            E[:, (vy % n)[:, None], (vx % n)[None, :]] = Kt[k] * W
            inten += st[k] * (torch.fft.ifft2(E) * (n * n)).abs() ** 2
        grid = torch.fft.fftshift(inten, dim=(1, 2))
        S = torch.fft.fft2(inten) / (n * n)
        full = torch.zeros(m.shape[0], Fy, Fx, dtype=torch.complex128, device=DEV)
        full[:, (by % Fy)[:, None], (bx % Fx)[None, :]] = S[:, (by % n)[:, None], (bx % n)[None, :]]
        img = torch.fft.fftshift(torch.fft.ifft2(full).real * (Fx * Fy), dim=(1, 2))
        out[b:b + step] = img[:, oy:oy + h, ox:ox + w] if crop else img
    return (out, torch.fft.fftshift(spec, dim=(1, 2)), grid) if conv else out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("image", "host"):
        K, s, Nx, Ny = kernels(pow2(case["Lx"]), pow2(case["Ly"]), case["nk"])
        return aerial(layouts(seed, case["B"], case["Ly"], case["Lx"], case["grey"]), K, s, Nx, Ny)
    if kind == "plan":
        out = []
        for s, n in sizes_of(case):
            p = 1024 if s <= 1024 else 2048
            K, sc, Nx, Ny = kernels(p, p, case["nk"])
            out += list(aerial(layouts(seed, n, s, s), K, sc, Nx, Ny, p, p, crop=False))
        return out
    if kind == "calls":
        K, s, Nx, Ny = kernels(pow2(case["Lx"]), pow2(case["Ly"]), case["nk"])
        image, spec, grid = aerial(layouts(seed, 1, case["Ly"], case["Lx"], True), K, s, Nx, Ny, conv=128)
        return [spec[0].real, spec[0].imag, image[0], grid[0]]
    if kind == "optics":
        src, N, defocus = optics_of(case, seed)
        P, J = pupil(src, case["L"], case["L"], N, N, defocus)
        K, s = top_kernels(P, J, case["nk"])
        A = P * np.sqrt(J)
        return [A @ A.conj().T, s, s, aerial(layouts(seed, 1, case["L"], case["L"]), K, s, N, N)]
    masks = layouts(seed, case["B"], case["L"], case["L"])
    theta = torch.as_tensor(weights(seed)).to(DEV).double()
    K, s, Nx, Ny = kernels(case["L"], case["L"], 24)
    if kind == "grad":
        theta.requires_grad_(True)
        targets = aerial(masks, K, s, Nx, Ny).float().double()
        d = (network(theta, masks.double()) - targets).reshape(case["B"], -1)
        loss = (d.norm(dim=1) / targets.reshape(case["B"], -1).norm(dim=1)).mean()
        loss.backward()
        return [loss.detach(), theta.grad]
    with torch.no_grad():
        net = torch.cat([network(theta, masks[b:b + 16].double()) for b in range(0, case["B"], 16)])
    L = case["L"]
    f = torch.fft.fftfreq(L, 1.0 / L, device=DEV).abs()
    spec = torch.fft.fft2(net) * ((f <= 2 * Ny)[:, None] & (f <= 2 * Nx)[None, :])
    return [torch.fft.ifft2(spec).real, None]
