"""The imaging stages behind litho_image_noalloc (csrc/imaging.cu, image_pipeline_noctx) on scratch memory that
holds anything at all: every region, the flag of the bounded waits among them, is written before it is
read.  Rows that go by bulk copies (a width that is no multiple of four) and rows that don't.
Held to the FP64 oracle at the imaging tolerance.
"""
import ctypes as C

import numpy as np
import pytest

from oracle import np_ref as R

pytestmark = pytest.mark.gpu

TOL = 1e-5


class ImgGeom(C.Structure):  # litho_internal.cuh
    _fields_ = [(n, C.c_int) for n in ("Lx", "Ly", "Fx", "Fy", "Nx", "Ny", "nk", "convN")]


class ImgPlan(C.Structure):
    _fields_ = [("g", ImgGeom)] + [(n, C.c_int) for n in ("batch", "rowBlocks", "colSplits", "kpg", "ngroups", "sms")] + [
        ("early", C.c_bool)]


@pytest.mark.parametrize("Lx,Ly", [(130, 121), (129, 64), (128, 121)])
@pytest.mark.parametrize("fill", [0xFF, 0x01])
def test_scratch_may_hold_anything(Lx, Ly, fill):
    import litho_gb300 as L
    import torch
    lib = L.lib()
    make_plan = getattr(lib, "_ZN5litho9make_planERKNS_7ImgGeomEii")
    make_plan.restype, make_plan.argtypes = ImgPlan, [C.POINTER(ImgGeom), C.c_int, C.c_int]
    layout = getattr(lib, "_ZN5litho20noctx_scratch_layoutERKNS_7ImgPlanEPm")
    layout.restype, layout.argtypes = C.c_size_t, [C.POINTER(ImgPlan), C.POINTER(C.c_size_t)]
    image = getattr(lib, "_ZN5litho20image_pipeline_noctxEP11CUstream_stRKNS_7ImgPlanEPKfS6_S6_S6_PcPf")
    image.restype, image.argtypes = C.c_int, [C.c_void_p, C.POINTER(ImgPlan)] + [C.c_void_p] * 6

    rng = np.random.default_rng(Lx + Ly)
    nx, ny, nk = 3, 4, 5
    n = (2 * nx + 1) * (2 * ny + 1)
    k = (rng.standard_normal((nk, n)) + 1j * rng.standard_normal((nk, n))).astype(np.complex64)
    s = rng.uniform(0.1, 1, nk).astype(np.float32)
    mask = (rng.random((Ly, Lx)) > 0.5).astype(np.float32)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dm, kr, ki, sc = up(mask), up(k.real), up(k.imag), up(s)
    geom = ImgGeom(Lx, Ly, L.next_pow2(Lx), L.next_pow2(Ly), nx, ny, nk, 32)
    plan = make_plan(C.byref(geom), 1, torch.cuda.get_device_properties(0).multi_processor_count)
    assert plan.batch == 1 and plan.g.Lx == Lx and plan.rowBlocks >= 1 and plan.ngroups >= 1
    scratch = torch.full((layout(C.byref(plan), (C.c_size_t * 8)()),), fill, dtype=torch.uint8, device="cuda")
    out = torch.full((Ly, Lx), float("nan"), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert image(stream, C.byref(plan), dm.data_ptr(), kr.data_ptr(), ki.data_ptr(), sc.data_ptr(), scratch.data_ptr(),
                 out.data_ptr()) == 0
    torch.cuda.synchronize()
    assert R.rel_l2(out.cpu().numpy(), R.mask_to_image(mask, k, s, nx, ny, conv_n=32, embed=None)) < TOL
