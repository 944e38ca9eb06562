"""Planes of 1024 rows, whose work planes are stored in the column tile's
swizzled order: widths whose rows take 4, 8, 16 and 32 lanes and the line
engine, every column width, against the FP64 oracle (RL parity tolerance of
1e-4 relative L2 on the estimate) and bit for bit among the column widths, for
few pairs and for many."""
import numpy as np
import pytest

from conftest import rel_l2
from gpu_deconvolution_b200 import api, synth
from oracle import fmvd_oracle as O

K = 9


@pytest.mark.gpu
@pytest.mark.parametrize("fftW", [16, 64, 256, 1024, 1536])
@pytest.mark.parametrize("bits", [16, 8])
def test_tall_planes(fftW, bits):
    import torch
    H, W, V, D = 1024 - K + 1, fftW - K + 1, 2, 9
    rng = np.random.default_rng(fftW + bits)
    views = rng.integers(10, 3000 if bits == 16 else 250, (V, D, H, W)).astype(np.uint16 if bits == 16 else np.uint8)
    w = [rng.uniform(0.3, 1.5, (H, W)).astype(np.float32) for _ in range(V)]
    psfs = [synth.gaussian_psf(K, K, 1.0, 2.0, 40.0 * v) for v in range(V)]
    t = torch.from_numpy(views.view(np.int16) if bits == 16 else views).cuda()
    res = []
    for planes in (D, 1):
        for cw in (0, 2, 4, 8):
            plan = api.DevicePlan(H, W, w, [p.copy() for p in psfs], 0, bits, col_warps=cw)
            try:
                assert (plan.fftH, plan.fftW) == (1024, fftW)
                out = torch.zeros((planes, H, W), dtype=t.dtype, device="cuda")
                est = torch.zeros((planes, 1024, fftW), dtype=torch.float32, device="cuda")
                plan.run(t[:, :planes].contiguous(), out, 3, estimate=est)
                torch.cuda.synchronize()
                res.append((out[:1].clone(), est[:1].clone()))
                assert plan.lib.fmvd_b200_plan_check(plan.plan) == 0
            finally:
                plan.destroy()
            if cw == 0 and planes == D:
                _, ref = O.deconvolve_volume(views[:, [0, D - 1]], w, psfs, 0, 3, bits=bits, return_float=True)
                assert rel_l2(est[[0, D - 1]].cpu().numpy(), ref) < 1e-4
    # one plane and nine may share a pair with another plane, which changes no
    # plane's bits beyond FP32 rounding; within a plane count the widths agree
    for group in (res[:4], res[4:]):
        assert all(torch.equal(group[0][0], o) and torch.equal(group[0][1], e) for o, e in group[1:])
