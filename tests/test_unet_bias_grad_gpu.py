"""The weight-gradient kernel's bias sums, which come from its staged tiles (one
swizzle for 32-channel tiles, another for 64, two tiles side by side for 128) by
two warps that release the stages with the MMAs, against FP64 sums, with the
weight gradient beside them; partial tiles, several CTAs, several output
tiles, images narrower than a tile.  The kernel is called through its internal
entry: the exported one asks for no bias gradient.

Tolerance: FP32 additions of bf16 values, 16 units of 2^-24 of the sum of their
magnitudes; a dropped or doubled pixel is some hundreds of times that."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_l2
from oracle import unet_oracle as U

ENTRY = "_ZN4fmvd4unet10conv_wgradERKNS0_9WgradDescEP11CUstream_st"


class WgradDesc(C.Structure):
    _fields_ = [("grad", C.c_void_p), ("in_", C.c_void_p)] + \
        [(n, C.c_int) for n in ("N", "H", "W", "cin", "cout", "taps")] + \
        [("dw", C.c_void_p), ("db", C.c_void_p), ("status", C.c_void_p)]


@pytest.mark.gpu
@pytest.mark.parametrize("cin,cout", [(32, 32), (32, 64), (32, 128), (32, 192), (64, 32), (64, 64), (64, 128),
                                      (128, 32), (256, 64)])
@pytest.mark.parametrize("N,H,W,taps", [(1, 8, 8, 9), (3, 12, 16, 9), (1, 34, 64, 9), (1, 136, 64, 1), (1, 16, 4, 9),
                                        (2, 72, 128, 9)])
def test_bias_sums(cin, cout, N, H, W, taps):
    import torch
    from gpu_deconvolution_b200 import native
    lib = native.load()
    fn = getattr(lib, ENTRY)
    fn.restype, fn.argtypes = C.c_bool, [C.POINTER(WgradDesc), C.c_void_p]
    g = torch.Generator(device="cuda").manual_seed(cin + cout + H)
    grad = torch.randn((N, H, W, cout), generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn((N, H, W, cin), generator=g, device="cuda").to(torch.bfloat16)
    dw = torch.zeros((cout, taps, cin), dtype=torch.float32, device="cuda")
    db = torch.full((cout,), 3.0, dtype=torch.float32, device="cuda")  # added to, not overwritten
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    native.clear_errors()
    d = WgradDesc(grad.data_ptr(), x.data_ptr(), N, H, W, cin, cout, taps, dw.data_ptr(), db.data_ptr(),
                  status.data_ptr())
    ok = fn(C.byref(d), None)
    native.check("conv_wgrad")
    assert ok
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    flat = grad.double().reshape(-1, cout)
    ref, size = flat.sum(0) + 3.0, flat.abs().sum(0) + 3.0
    assert bool(((db.double() - ref).abs() <= 16 * 2.0 ** -24 * size).all())
    ref = U.conv_wgrad(grad.float().cpu().numpy(), x.float().cpu().numpy(), taps)
    assert rel_l2(dw.cpu().numpy(), ref) < 2e-5  # as for the weight gradient's other tests
    assert np.isfinite(dw.cpu().numpy()).all()
