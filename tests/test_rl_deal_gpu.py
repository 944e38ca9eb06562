"""Which runs are dealt over the two lanes: one lane while the column pass of all
pairs is resident on the multiprocessors at once (seen in the launch count), and
the same planes and estimates bit for bit on either side of the line, from a
given first estimate and inside a captured batch too."""
import numpy as np
import pytest

from gpu_deconvolution_b200 import api, native, synth

K, V = 9, 2


def _plan(fft, **kw):
    h, w = fft[0] - K + 1, fft[1] - K + 1
    rng = np.random.default_rng(fft[0] + fft[1])
    ws = [rng.uniform(0.3, 1.5, (h, w)).astype(np.float32) for _ in range(V)]
    plan = api.DevicePlan(h, w, ws, [synth.gaussian_psf(K, K, 1.2, 2.5, 40.0 * v) for v in range(V)], 0, **kw)
    assert (plan.fftH, plan.fftW) == fft
    return plan


def _views(torch, plan, planes):
    g = torch.Generator(device="cuda").manual_seed(planes)
    return torch.randint(20, 3000, (V, planes, plan.dataH, plan.dataW), generator=g, device="cuda").to(torch.int16)


@pytest.mark.gpu
@pytest.mark.parametrize("fft,pairs,batches", [((1024, 64), 33, 1), ((1024, 64), 37, 1), ((1024, 64), 38, 2),
                                               ((512, 256), 18, 1), ((512, 256), 19, 2), ((1536, 64), 27, 1),
                                               ((1536, 64), 28, 2), ((2560, 64), 18, 1), ((2560, 64), 19, 2),
                                               ((4096, 128), 4, 1), ((4096, 128), 5, 2)])
def test_line_of_the_deal(fft, pairs, batches):
    import torch
    planes = 2 * pairs - 1
    lib = native.load()
    res = []
    for ppb in (0, 1):
        plan = _plan(fft, pairs_per_batch=ppb)
        try:
            views = _views(torch, plan, planes)
            out = torch.zeros((planes, plan.dataH, plan.dataW), dtype=torch.int16, device="cuda")
            est = torch.zeros((planes, *fft), dtype=torch.float32, device="cuda")
            init = torch.full_like(est, 500.0) + 100.0 * torch.arange(planes, device="cuda")[:, None, None]
            n0 = lib.fmvd_b200_launch_count()
            plan.run(views, out, 2, estimate=est, init=init)
            launches = lib.fmvd_b200_launch_count() - n0
            torch.cuda.synchronize()
            # per batch: the first pass, four per view update and the estimate's write-out
            per_batch = 1 + 4 * V * 2 + 1
            assert launches == (batches if ppb == 0 else pairs) * per_batch
            res.append((out, est))
        finally:
            plan.destroy()
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


@pytest.mark.gpu
def test_dealt_runs_in_a_captured_batch():
    import torch
    plans = [_plan((512, 256)), _plan((1536, 64))]
    try:
        views = [_views(torch, p, n) for p, n in zip(plans, (41, 60))]
        outs = [torch.zeros((v.shape[1], p.dataH, p.dataW), dtype=torch.int16, device="cuda")
                for p, v in zip(plans, views)]
        refs = [torch.zeros_like(o) for o in outs]
        for p, v, r in zip(plans, views, refs):
            p.run(v, r, 3)
        torch.cuda.synchronize()
        batch = api.Batch(plans, views, outs, 3, max_branches=2)
        try:
            for _ in range(2):
                for o in outs:
                    o.zero_()
                torch.cuda.synchronize()
                batch.run()
                torch.cuda.synchronize()
                assert all(torch.equal(o, r) for o, r in zip(outs, refs))
        finally:
            batch.destroy()
    finally:
        for p in plans:
            p.destroy()
