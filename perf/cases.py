"""Performance cases of the reconstruction framework: what a user's program has
it do, through the public entry points, with inputs made from a seed.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same
ranges, ``prepare`` builds what a program holds before the call, ``run`` is one
pass, ``work`` the bytes and operations a pass cannot do without, and ``exact``
the result in 64 bits from plain torch where one exists.
"""
import math

import numpy as np
import torch

from gpu_deconvolution_b200 import api, synth
from gpu_deconvolution_b200.warmstart import WarmStartNet

DEV = "cuda"


def listed():
    return [
        # a preview of a small region of interest: launches and latency count
        rl("rl_128_call", 2, 4, 128, 128, 9, 9, 10),
        # the small plain-RL workload (two views of a 256 x 256 x 64 bead
        # field, 17 x 17 PSFs), with the float estimate a later stage continues
        rl("rl_256_volume", 2, 64, 256, 256, 17, 17, 10, estimate=True),
        # the headline workload: a 512 x 512 x 384 frame, four views, 20 iterations
        rl("rl_512_volume", 4, 384, 512, 512, 31, 31, 20),
        # 8-bit camera crops of odd size and an odd plane count, continued from
        # an earlier estimate as the convergence check does
        rl("rl_ragged_8bit", 3, 15, 333, 477, 21, 13, 8, bits=8, psf_type=3, estimate=True, init=True),
        # full camera frames that need an FFT plane of 1536 x 1536
        rl("rl_1400", 4, 12, 1400, 1400, 63, 63, 10, psf_type=1),
        # the large streamed workload's planes (six views, FFT plane 2560 x
        # 2560), odd plane count
        rl("rl_2048", 6, 5, 2048, 2048, 63, 63, 5, estimate=True),
        # the four rotated views of the headline workload into the common frame
        resample("resample_rotated", 4, (128, 512, 512), (384, 512, 512), 16, 3.0, 0.0, False),
        # views with registration matrices (small shears and scales on top of
        # the rotation), 8 bit, odd sizes, samples and the float frame
        resample("resample_registered_8bit", 3, (97, 271, 333), (251, 355, 402), 8, 2.5, 0.02, True),
        # host volumes in, reconstructed host volume out, plan kept
        reconstruct("reconstruct_host", 4, (96, 320, 400), (200, 320, 400), 31, 10, 2.0),
        # the drop-in streaming interface with C callbacks over host planes,
        # plan made and released inside, as a caller of the C API does
        stream("stream_host", 3, 24, 300, 420, 17, 10),
        # learned warm start: network estimate of 64 planes of four views
        unet("unet_forward", 4, 64, 512, 512, 16, False),
        # one training step of the same network at its batch of 16
        unet("unet_train", 4, 16, 512, 512, 16, True),
    ]


# ------------------------------------------------------------------ the kinds
def rl(name, views, planes, h, w, kh, kw, iterations, bits=16, psf_type=0, estimate=False, init=False):
    return {"name": name, "kind": "rl", "views": views, "planes": planes, "h": h, "w": w, "kh": kh, "kw": kw,
            "iterations": iterations, "bits": bits, "psf_type": psf_type, "estimate": estimate, "init": init}


def resample(name, views, src, frame, bits, zscale, shear, float_frame):
    return {"name": name, "kind": "resample", "views": views, "d": src[0], "h": src[1], "w": src[2], "td": frame[0],
            "th": frame[1], "tw": frame[2], "bits": bits, "zscale": zscale, "shear": shear,
            "float_frame": float_frame}


def reconstruct(name, views, src, frame, k, iterations, zscale):
    return {"name": name, "kind": "reconstruct", "views": views, "d": src[0], "h": src[1], "w": src[2],
            "td": frame[0], "th": frame[1], "tw": frame[2], "k": k, "iterations": iterations, "zscale": zscale}


def stream(name, views, planes, h, w, k, iterations):
    return {"name": name, "kind": "stream", "views": views, "planes": planes, "h": h, "w": w, "k": k,
            "iterations": iterations}


def unet(name, views, planes, h, w, batch, train):
    return {"name": name, "kind": "unet", "views": views, "planes": planes, "h": h, "w": w, "batch": batch,
            "train": train}


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rl", "rl", "rl", "resample", "resample", "reconstruct", "stream", "unet"])
    if kind == "rl":
        h, w = log_int(rng, 96, 2048), log_int(rng, 96, 2048)
        kmax = min(63, h // 4, w // 4)
        kh, kw = (2 * (log_int(rng, 7, kmax) // 2) + 1 for _ in range(2))
        views, iterations = rng.randint(2, 6), rng.randint(3, 20)
        per_plane = fft_size(h + kh - 1) * fft_size(w + kw - 1) * views * iterations
        planes = max(1, min(log_int(rng, 1, 128), int(5e9 / per_plane)))
        c = rl("", views, planes, h, w, kh, kw, iterations, rng.choice([8, 16]), rng.choice([0, 1, 3]),
               rng.random() < 0.5, rng.random() < 0.3)
    elif kind == "resample":
        src = (log_int(rng, 16, 160), log_int(rng, 100, 640), log_int(rng, 100, 640))
        frame = (log_int(rng, 16, 320), log_int(rng, 100, 640), log_int(rng, 100, 640))
        c = resample("", rng.randint(1, 6), src, frame, rng.choice([8, 16]), rng.uniform(1.0, 4.0),
                     rng.choice([0.0, rng.uniform(0.001, 0.05)]), rng.random() < 0.3)
    elif kind == "reconstruct":
        h, w = log_int(rng, 100, 480), log_int(rng, 100, 480)
        d, z = log_int(rng, 16, 128), rng.uniform(1.0, 3.0)
        c = reconstruct("", rng.randint(2, 5), (d, h, w), (int(d * z), h, w), rng.choice([9, 17, 31]),
                        rng.randint(3, 12), z)
    elif kind == "stream":
        c = stream("", rng.randint(2, 5), log_int(rng, 2, 64), log_int(rng, 100, 480), log_int(rng, 100, 480),
                   rng.choice([9, 17, 31]), rng.randint(3, 12))
    else:
        train = rng.random() < 0.5
        c = unet("", rng.randint(1, 6), rng.randint(1, 16) if train else log_int(rng, 1, 64),
                 64 * rng.randint(2, 8), rng.choice([128, 256, 512]), 16, train)
    del c["name"]
    return c


# --------------------------------------------------------------------- inputs
def fft_size(n):
    """Length the reference pads to: a multiple of 16, then the next power of
    two up to 1024, then the next multiple of 512."""
    n = -(-n // 16) * 16
    p = 1 << (n - 1).bit_length()
    return p if p <= 1024 else -(-n // 512) * 512


def psfs(views, kh, kw):
    s = min(5.0, max(1.2, min(kh, kw) / 6.0))
    return [synth.gaussian_psf(kh, kw, 1.2, s, 180.0 * v / views) for v in range(views)]


def weights(views, h, w):
    """Per-view weight planes falling off smoothly from a view's own side."""
    y = np.linspace(0.0, 1.0, h, dtype=np.float32)[:, None]
    x = np.linspace(0.0, 1.0, w, dtype=np.float32)[None, :]
    out = []
    for v in range(views):
        a = 2.0 * np.pi * v / views
        out.append((0.6 + 0.4 * np.sin(a + 2.0 * x) * np.cos(a - y)).astype(np.float32))
    return out


def bead_views(c, seed, kernels, bits):
    """views x planes x h x w samples: beads on a background, blurred with each
    view's PSF, with photon noise."""
    gt, g = synth.bead_volume_torch(c["planes"], c["h"], c["w"], seed, DEV, 2e-4)
    if bits == 8:
        gt = gt * (200.0 / float(gt.max()))
    return synth.blur_noise_torch(gt, kernels, g, bits)


def pad_index(n, size, border):
    """Source index of each padded position: clamped within ``border`` past the
    end, 0 beyond."""
    i = torch.arange(size, device=DEV)
    return torch.where(i < n + border, i.clamp(max=n - 1), torch.zeros_like(i))


def samples(t, bits):
    """Integer samples as float64 (16-bit samples are held as int16 bits)."""
    return (t.to(torch.int32) & (0xFFFF if bits == 16 else 0xFF)).to(torch.float64)


def matrices(c, seed):
    r = np.random.default_rng(seed)
    frame, src = (c["td"], c["th"], c["tw"]), (c["d"], c["h"], c["w"])
    out = []
    for v in range(c["views"]):
        m = synth.rotation_y_inverse(360.0 * v / c["views"], frame, src, c["zscale"], r.uniform(-8.0, 8.0, 3))
        m = m.reshape(3, 4).astype(np.float64)
        e = np.eye(3) + c.get("shear", 0.0) * r.uniform(-1.0, 1.0, (3, 3))
        centre = np.array([c["tw"], c["th"], c["td"]]) / 2.0
        m = np.concatenate([m[:, :3] @ e, (m[:, 3] + m[:, :3] @ (centre - e @ centre))[:, None]], axis=1)
        out.append(np.ascontiguousarray(m.astype(np.float32).reshape(12)))
    return out


def source_volumes(c, seed, bits):
    gt, g = synth.bead_volume_torch(c["d"], c["h"], c["w"], seed, DEV, 2e-4)
    if bits == 8:
        gt = gt * (200.0 / float(gt.max()))
    v = [torch.poisson(gt, generator=g).round() for _ in range(c["views"])]
    return torch.stack([x.to(torch.int32).to(torch.int16) if bits == 16 else x.to(torch.uint8) for x in v])


def unet_layers():
    """(cin, cout, taps) of the network's convolutions, in parameter order."""
    b = 32
    out = [(64, b, 1), (b, b, 9)]
    for n in range(1, 4):
        out += [(b << (n - 1), b << n, 9), (b << n, b << n, 9)]
    for n in (2, 1, 0):
        out += [(b << (n + 1), b << n, 9), (b << n, b << n, 9)]
    return out


def unet_params(views, seed):
    """Weights of the size a trained network has (He-scaled, small biases)."""
    r = np.random.default_rng(seed)
    parts = []
    for i, (cin, cout, taps) in enumerate(unet_layers()):
        fan = 9 * (views + 1) if i == 0 else taps * cin
        w = r.standard_normal((cout, taps, cin), dtype=np.float32) * np.float32(math.sqrt(2.0 / fan))
        if i == 0:
            w[:, :, 9 * (views + 1):] = 0.0
        parts += [w.reshape(-1), 0.01 * r.standard_normal(cout, dtype=np.float32)]
    parts += [0.05 * r.standard_normal(32, dtype=np.float32), np.ones(1, np.float32)]
    return np.concatenate(parts)


def unet_inputs(c, seed):
    kernels = [synth.gaussian_psf(17, 17, 1.5, 4.0, 180.0 * v / c["views"]) for v in range(c["views"])]
    gt, g = synth.bead_volume_torch(c["planes"], c["h"], c["w"], seed, DEV, 5e-5)
    return synth.blur_noise_torch(gt, kernels, g, 16), gt.contiguous()


# -------------------------------------------------------------------- prepare
def prepare(case, seed):
    return {"rl": prepare_rl, "resample": prepare_resample, "reconstruct": prepare_reconstruct,
            "stream": prepare_stream, "unet": prepare_unet}[case["kind"]](case, seed)


def prepare_rl(c, seed):
    k = psfs(c["views"], c["kh"], c["kw"])
    views = bead_views(c, seed, k, c["bits"])
    plan = api.DevicePlan(c["h"], c["w"], weights(c["views"], c["h"], c["w"]), [p.copy() for p in k], c["psf_type"],
                          c["bits"])
    out = torch.empty((c["planes"], c["h"], c["w"]), dtype=views.dtype, device=DEV)
    est = init = None
    if c["estimate"]:
        est = torch.empty((c["planes"], plan.fftH, plan.fftW), dtype=torch.float32, device=DEV)
    if c["init"]:
        init = start_estimate(c, views, plan.fftH, plan.fftW).to(torch.float32).contiguous()
    return {"case": c, "plan": plan, "views": views, "out": out, "est": est, "init": init}


def start_estimate(c, views, fh, fw):
    """The views' mean on the padded plane, an estimate RL can go on from."""
    mean = sum(samples(v, c["bits"]) for v in views) / c["views"] + 1.0
    y = pad_index(c["h"], fh, c["kh"] // 2)
    x = pad_index(c["w"], fw, c["kw"] // 2)
    return mean[:, y][:, :, x]


def prepare_resample(c, seed):
    vols = source_volumes(c, seed, c["bits"])
    pitch = api.source_pitch(c["bits"], c["w"])
    src = torch.zeros((c["views"], c["d"], c["h"], pitch), dtype=vols.dtype, device=DEV)
    src[..., :c["w"]] = vols
    shape = (c["views"], c["td"], c["th"], c["tw"])
    out = torch.empty(shape, dtype=vols.dtype, device=DEV)
    frame = torch.empty(shape, dtype=torch.float32, device=DEV) if c["float_frame"] else None
    return {"case": c, "src": src, "pitch": pitch, "m": matrices(c, seed), "out": out, "frame": frame}


def prepare_reconstruct(c, seed):
    k = psfs(c["views"], c["k"], c["k"])
    plan = api.DevicePlan(c["th"], c["tw"], weights(c["views"], c["th"], c["tw"]), [p.copy() for p in k], 0, 16)
    rec = api.Reconstructor(plan, c["views"], (c["d"], c["h"], c["w"]), (c["td"], c["th"], c["tw"]))
    host = [v.cpu().pin_memory().numpy().view(np.uint16) for v in source_volumes(c, seed, 16)]
    out = torch.empty((c["td"], c["th"], c["tw"]), dtype=torch.int16).pin_memory().numpy().view(np.uint16)
    return {"case": c, "plan": plan, "rec": rec, "host": host, "out": out, "m": matrices(c, seed)}


def prepare_stream(c, seed):
    k = psfs(c["views"], c["k"], c["k"])
    views = bead_views(c, seed, k, 16).cpu().numpy().view(np.uint16)
    return {"case": c, "views": views, "weights": weights(c["views"], c["h"], c["w"]), "psfs": k}


def prepare_unet(c, seed):
    views, target = unet_inputs(c, seed)
    net = WarmStartNet(c["h"], c["w"], c["views"], max_batch=c["batch"], seed=0)
    net.set_params(unet_params(c["views"], seed))
    out = None if c["train"] else torch.empty((c["planes"], c["h"], c["w"]), dtype=torch.float32, device=DEV)
    return {"case": c, "net": net, "views": views, "target": target, "out": out}


# ------------------------------------------------------------------------ run
def run(state):
    c = state["case"]
    if c["kind"] == "rl":
        state["plan"].run(state["views"], state["out"], c["iterations"], estimate=state["est"], init=state["init"])
        return {"samples": state["out"], "estimate": state["est"]}
    if c["kind"] == "resample":
        for v in range(c["views"]):
            api.transform_device(state["src"][v], state["pitch"], c["w"], c["h"], c["d"], state["m"][v], c["tw"],
                                 c["th"], 0, c["td"], out=state["out"][v],
                                 out_f32=state["frame"][v] if state["frame"] is not None else None, bits=c["bits"])
        return {"samples": state["out"], "frame": state["frame"]}
    if c["kind"] == "reconstruct":
        return {"samples": state["rec"].run(state["host"], state["m"], c["iterations"], out=state["out"])}
    if c["kind"] == "stream":
        return {"samples": api.deconvolve_c_callbacks(state["views"], state["weights"], state["psfs"], 0,
                                                      c["iterations"])}
    if c["train"]:
        # the step size the cosine schedule ends on, scaled down so that the
        # same weights are met again by a repeated pass
        loss = state["net"].train_step(state["views"], state["target"], 1e-9)
        return {"loss": loss, "grads": state["net"].grads()}
    return {"estimate": state["net"].forward(state["views"], out=state["out"])}


# ----------------------------------------------------------------------- work
def rl_work(views, planes, h, w, kh, kw, iterations, es, estimate=False, init=False):
    fh, fw = fft_size(h + kh - 1), fft_size(w + kw - 1)
    per = 10.0 * fh * fw * math.log2(fh * fw) + 20.0 * fh * fw  # four real transforms and the element-wise steps
    b = planes * h * w * es * (views + 1) + 4 * views * h * w + 4 * planes * fh * fw * (int(estimate) + int(init))
    return {"bytes": b, "flops": planes * views * iterations * per}


def work(case):
    c = case
    if c["kind"] == "rl":
        return rl_work(c["views"], c["planes"], c["h"], c["w"], c["kh"], c["kw"], c["iterations"], c["bits"] // 8,
                       c["estimate"], c["init"])
    if c["kind"] == "resample":
        es, n = c["bits"] // 8, c["td"] * c["th"] * c["tw"]
        return {"bytes": c["views"] * (c["d"] * c["h"] * c["w"] * es + n * (es + (4 if c["float_frame"] else 0))),
                "flops": c["views"] * n * 45.0}
    if c["kind"] == "reconstruct":
        r = rl_work(c["views"], c["td"], c["th"], c["tw"], c["k"], c["k"], c["iterations"], 2)
        return {"bytes": 2 * c["views"] * c["d"] * c["h"] * c["w"] + 2 * c["td"] * c["th"] * c["tw"],
                "flops": r["flops"] + c["views"] * c["td"] * c["th"] * c["tw"] * 45.0}
    if c["kind"] == "stream":
        return rl_work(c["views"], c["planes"], c["h"], c["w"], c["k"], c["k"], c["iterations"], 2)
    px = c["planes"] * c["h"] * c["w"]
    level = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0]
    macs = sum(px / 4 ** n * cin * cout * taps for n, (cin, cout, taps) in zip(level, unet_layers()))
    n = sum(cin * cout * taps + cout for cin, cout, taps in unet_layers()) + 33
    return {"bytes": px * (2 * c["views"] + 4) + 4 * n * (2 if c["train"] else 1),
            "flops": 2.0 * macs * (3 if c["train"] else 1)}


# ---------------------------------------------------------------------- exact
def exact(case, seed):
    if case["kind"] == "rl" and case["estimate"] and case["psf_type"] in (0, 3):
        return exact_rl(case, seed)
    if case["kind"] == "resample" and case["float_frame"]:
        return exact_resample(case, seed)
    if case["kind"] == "unet":
        return exact_unet(case, seed)
    return None


def exact_rl(c, seed):
    """Multi-view Richardson-Lucy on the padded plane, float64."""
    k = psfs(c["views"], c["kh"], c["kw"])
    views = bead_views(c, seed, k, c["bits"])
    fh, fw = fft_size(c["h"] + c["kh"] - 1), fft_size(c["w"] + c["kw"] - 1)
    ws = [torch.from_numpy(w.astype(np.float64)).to(DEV) for w in weights(c["views"], c["h"], c["w"])]
    total = sum(ws)

    def spectrum(p):
        plane = torch.zeros((fh, fw), dtype=torch.float64, device=DEV)
        plane[:c["kh"], :c["kw"]] = torch.from_numpy(p / p.sum()).to(DEV)
        return torch.fft.rfft2(torch.roll(plane, (-(c["kh"] // 2), -(c["kw"] // 2)), (0, 1)))

    def padded(t, by, bx):
        return t[..., pad_index(c["h"], fh, by), :][..., pad_index(c["w"], fw, bx)]

    prepared = []
    for v in range(c["views"]):
        p = k[v].astype(np.float64)
        mirror = p[::-1, ::-1].copy()
        second = mirror if c["psf_type"] == 0 else mirror ** c["views"]
        # data is padded with the kernel's half sizes swapped, as the reference does
        prepared.append((spectrum(p), spectrum(second), padded(ws[v] / total, c["kh"] // 2, c["kw"] // 2)))
    first = start_estimate(c, views, fh, fw).to(torch.float32).to(torch.float64) if c["init"] else None
    est = torch.empty((c["planes"], fh, fw), dtype=torch.float64, device=DEV)
    for z0 in range(0, c["planes"], 8):
        n = min(8, c["planes"] - z0)
        e = first[z0:z0 + n] if first is not None else torch.full((n, fh, fw), 10.0 * c["views"],
                                                                 dtype=torch.float64, device=DEV)
        for _ in range(c["iterations"]):
            for v, (s1, s2, w) in enumerate(prepared):
                blur = torch.fft.irfft2(torch.fft.rfft2(e) * s1, s=(fh, fw))
                d = padded(samples(views[v, z0:z0 + n], c["bits"]), c["kw"] // 2, c["kh"] // 2)
                ratio = torch.where(blur > 1.0, d / blur, blur)
                r = torch.fft.irfft2(torch.fft.rfft2(ratio) * s2, s=(fh, fw))
                e = e + w * (e * r - e)
        est[z0:z0 + n] = e
    return {"samples": None, "estimate": est}


def exact_resample(c, seed):
    """Trilinear interpolation with texture-style 1/256 weights, float64."""
    vols = source_volumes(c, seed, c["bits"])
    frame = torch.empty((c["views"], c["td"], c["th"], c["tw"]), dtype=torch.float64, device=DEV)
    x = torch.arange(c["tw"], device=DEV, dtype=torch.float64)[None, None, :]
    y = torch.arange(c["th"], device=DEV, dtype=torch.float64)[None, :, None]
    size = (c["w"], c["h"], c["d"])
    for v, m in enumerate(matrices(c, seed)):
        m = m.reshape(3, 4).astype(np.float64)
        vol = samples(vols[v], c["bits"])
        for z0 in range(0, c["td"], 32):
            z = torch.arange(z0, min(z0 + 32, c["td"]), device=DEV, dtype=torch.float64)[:, None, None]
            index, weight = [], []
            for a in range(3):
                q = torch.floor((m[a, 0] * x + m[a, 1] * y + m[a, 2] * z + m[a, 3]) * 256.0 + 0.5)
                index.append(torch.floor(q / 256.0).to(torch.int64))
                weight.append(q / 256.0 - torch.floor(q / 256.0))
            acc = 0.0
            for corner in range(8):
                inside, at, w = True, [], 1.0
                for a in range(3):
                    o = (corner >> a) & 1
                    i = index[a] + o
                    inside = (i >= 0) & (i < size[a]) & inside
                    at.append(i.clamp(0, size[a] - 1))
                    w = w * (weight[a] if o else 1.0 - weight[a])
                acc = acc + torch.where(inside, vol[at[2], at[1], at[0]], torch.zeros((), dtype=torch.float64,
                                                                                     device=DEV)) * w
            frame[v, z0:z0 + z.shape[0]] = acc
    return {"samples": None, "frame": frame}


def exact_unet(c, seed):
    """The network in float64 (no rounding of weights or activations)."""
    views, target = unet_inputs(c, seed)
    V = c["views"]
    flat = torch.from_numpy(unet_params(V, seed)).to(DEV).to(torch.float64)
    flat.requires_grad_(c["train"])
    layers, at = [], 0
    for cin, cout, taps in unet_layers():
        w = flat[at:at + cout * taps * cin].view(cout, taps, cin)
        at += cout * taps * cin
        layers.append((w, flat[at:at + cout]))
        at += cout
    out_w, out_b = flat[at:at + 32], flat[at + 32]

    def conv(i, x):
        w, b = layers[i]
        if i == 0:  # 3 x 3 patches of the views and their mean, tap-major
            w = w[:, 0, :9 * (V + 1)].reshape(32, 9, V + 1)
        k = w.permute(0, 2, 1).reshape(w.shape[0], w.shape[2], 3, 3)
        p = torch.nn.functional.pad(x, (1, 1, 1, 1))
        h, wd = x.shape[2], x.shape[3]
        acc = b.view(1, -1, 1, 1)
        for dy in range(3):
            for dx in range(3):
                acc = acc + torch.einsum("oc,nchw->nohw", k[:, :, dy, dx], p[:, :, dy:dy + h, dx:dx + wd])
        return acc

    def network(x):
        relu, up, pool = torch.relu, (lambda t: t.repeat_interleave(2, 2).repeat_interleave(2, 3)), \
            (lambda t: torch.nn.functional.avg_pool2d(t, 2))
        enc = []
        for n in range(4):
            x = relu(conv(2 * n, x if n == 0 else pool(x)))
            x = relu(conv(2 * n + 1, x))
            enc.append(x)
        for i, n in zip((8, 10, 12), (2, 1, 0)):
            x = relu(conv(i, up(x)) + enc[n])
            x = relu(conv(i + 1, x))
        return (x * out_w.view(1, -1, 1, 1)).sum(1) + out_b

    est = torch.empty((c["planes"], c["h"], c["w"]), dtype=torch.float64, device=DEV)
    loss = 0.0
    step = 2 if c["train"] else 4
    for z0 in range(0, c["planes"], step):
        v = samples(views[:, z0:z0 + step], 16)
        s = 1.0 + v.mean(dim=(0, 2, 3))
        x = torch.cat([v, v.mean(0, keepdim=True)]).permute(1, 0, 2, 3) / s.view(-1, 1, 1, 1)
        if c["train"]:
            t = target[z0:z0 + step].to(torch.float64) / s.view(-1, 1, 1)
            part = (network(x) - t).abs().sum() / float(c["planes"] * c["h"] * c["w"])
            part.backward()
            loss += float(part.detach())
        else:
            est[z0:z0 + step] = network(x) * s.view(-1, 1, 1)
    if c["train"]:
        return {"loss": loss, "grads": flat.grad.cpu().numpy()}
    return {"estimate": est}
