"""Convolution GEMMs at the edges of their tiles, against the FP64 oracle:
every layer shape of the border-tile forward kernel and of the all-taps weight
gradient, at heights that are not whole tiles, the narrowest width, several
tiles per CTA, and operands off a 16-byte boundary."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import unet_oracle as U

# FP32 accumulation over at most 9 * 256 products or 64 * 136 pixels: a few
# times 1e-7 for rounding, 1e-9 per accumulated pixel for the tensor cores'
# rounding towards zero
TOL = 2e-5


def _bf(torch, shape, g, scale=1.0):
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


def _np(t):
    return t.float().cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("cin,cout", [(32, 16), (32, 32), (32, 64), (32, 128), (64, 16), (64, 32), (64, 64),
                                      (64, 128), (128, 32), (128, 64)])
@pytest.mark.parametrize("N,H,W", [(1, 16, 8), (2, 24, 16), (1, 17, 128)])
def test_border_tile_forward(cin, cout, N, H, W):
    import torch
    from gpu_deconvolution_b200 import native
    lib = native.load()
    g = torch.Generator(device="cuda").manual_seed(cin + cout + H)
    x, w = _bf(torch, (N, H, W, cin), g), _bf(torch, (cout, 9, cin), g, 0.1)
    # skip and mask tensors two bytes off a 16-byte boundary in one of the runs
    for shift in (0, 1):
        add = _bf(torch, (N * H * W * cout + shift,), g)[shift:]
        mask = _bf(torch, (N * H * W * cout + shift,), g)[shift:]
        bias = torch.randn(cout + shift, generator=g, device="cuda")[shift:]
        outf = torch.zeros((N, H, W, cout), dtype=torch.float32, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        native.clear_errors()
        r = lib.fmvd_b200_conv_bf16(x.data_ptr(), w.data_ptr(), N, H, W, cin, cout, 9, None, outf.data_ptr(),
                                    bias.data_ptr(), add.data_ptr(), mask.data_ptr(), 1, status.data_ptr(), None)
        native.check("fmvd_b200_conv_bf16")
        assert r == 0
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        ref = U.conv(_np(x), _np(w), _np(bias), _np(add).reshape(outf.shape), True, _np(mask).reshape(outf.shape))
        assert rel_l2(_np(outf), ref) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("cin,cout", [(32, 32), (32, 64), (32, 128), (32, 192), (64, 32), (64, 64), (64, 192),
                                      (128, 32), (128, 64), (256, 32), (512, 64)])
@pytest.mark.parametrize("N,H,W,taps", [(1, 8, 8, 9), (3, 12, 16, 9), (1, 34, 64, 9), (1, 8, 8, 1), (1, 136, 64, 1)])
def test_all_taps_weight_gradient(cin, cout, N, H, W, taps):
    import torch
    from gpu_deconvolution_b200 import native
    lib = native.load()
    g = torch.Generator(device="cuda").manual_seed(cin + cout + H)
    grad, x = _bf(torch, (N, H, W, cout), g), _bf(torch, (N, H, W, cin), g)
    dw = torch.ones((cout, taps, cin), dtype=torch.float32, device="cuda")  # added to, not overwritten
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    native.clear_errors()
    r = lib.fmvd_b200_conv_wgrad_bf16(grad.data_ptr(), x.data_ptr(), N, H, W, cin, cout, taps, dw.data_ptr(),
                                      status.data_ptr(), None)
    native.check("fmvd_b200_conv_wgrad_bf16")
    assert r == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert rel_l2(dw.cpu().numpy(), 1.0 + U.conv_wgrad(_np(grad), _np(x), taps)) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("V,N,H,W", [(1, 1, 128, 128), (6, 2, 192, 256)])
def test_network_input_patches_and_output_gradient(V, N, H, W):
    """One to six views (patch rows of 18 to 63 values) and a height that is
    not a multiple of the coarsest level's tile."""
    import torch
    from gpu_deconvolution_b200.warmstart import WarmStartNet
    net = WarmStartNet(H, W, V, max_batch=N, seed=4)
    try:
        rng = np.random.default_rng(V)
        views_np = rng.integers(100, 2000, (V, N, H, W)).astype(np.uint16)
        target_np = rng.uniform(100, 2000, (N, H, W)).astype(np.float32)
        views = torch.from_numpy(views_np.view(np.int16)).cuda()
        p = net.params()
        est = net.forward(views)
        torch.cuda.synchronize()
        # bf16 storage between the layers, as for the network's other sizes
        assert rel_l2(est.cpu().numpy(), U.network_forward(p, views_np)[0]) < 1e-2
        loss = net.train_step(views, torch.from_numpy(target_np).cuda(), 0.0)
        ref_loss, ref_g = U.network_grads(p, views_np, target_np)
        assert abs(loss - ref_loss) < 1e-3 * ref_loss
        g = net.grads()
        off = 0
        for cin, cout, taps in U.layer_shapes(V):
            n = cout * taps * cin
            assert rel_l2(g[off:off + n], ref_g[off:off + n]) < 5e-2
            assert rel_l2(g[off + n:off + n + cout], ref_g[off + n:off + n + cout]) < 5e-2
            off += n + cout
        assert rel_l2(g[off:], ref_g[off:]) < 1e-2
        net.check()
    finally:
        net.destroy()
