"""The even split of a run over the two lanes: plane counts on both sides of
its threshold and with remainders give the planes and estimates of one pair
per batch, bit for bit; a batch size of the caller's is kept."""
import numpy as np
import pytest

from gpu_deconvolution_b200 import api, synth


@pytest.mark.gpu
@pytest.mark.parametrize("n,planes", [(470, 15), (470, 17), (470, 24), (470, 51), (1000, 3), (1000, 5), (1000, 13),
                                      (240, 67), (1100, 5)])
def test_even_split_equals_single_pairs(n, planes):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n + planes)
    views = torch.randint(0, 3000, (2, planes, n, n), generator=g, device="cuda").to(torch.int16)
    w = [(0.2 + np.random.default_rng(v).random((n, n))).astype(np.float32) for v in range(2)]
    res = []
    for pairs in (0, 1):
        psfs = [synth.gaussian_psf(9, 11, 1.2, 2.5, 40.0 * v) for v in range(2)]
        plan = api.DevicePlan(n, n, w, psfs, 0, 16, pairs_per_batch=pairs)
        assert pairs == 0 or plan.pairs_per_batch == pairs
        out = torch.zeros((planes, n, n), dtype=torch.int16, device="cuda")
        est = torch.zeros((planes, plan.fftH, plan.fftW), dtype=torch.float32, device="cuda")
        plan.run(views, out, 2, estimate=est)
        torch.cuda.synchronize()
        res.append((out, est))
        plan.destroy()
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
