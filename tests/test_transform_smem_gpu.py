"""Resampler launches whose brick is just below 48 KB: with the kernel's static
shared memory they pass the limit of a launch without an opt-in.  The first
call of a process has to have it, whatever the brick sizes of other calls, so
every map runs first in a process of its own.  Samples against the CPU oracle,
equal up to the final rounding as in the resampler's other tests; the
coefficients are multiples of 2^-10, so that every coordinate is exact."""
import math
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from oracle import fmvd_oracle as O

SRC, FRAME = (19, 50, 61), (17, 40, 45)  # d, h, w; td, th, tw


def _about_y(angle, scale, zscale):
    c, s = math.cos(math.radians(angle)), math.sin(math.radians(angle))
    return np.array([[scale * c, 0, scale * s], [0, scale, 0], [-scale * s / zscale, 0, scale * c / zscale]])


MAPS = {  # bits, linear part, tile (x, y, z), brick bytes
    "about_y_1.3": (8, _about_y(0, 1.3, 1.2), (32, 32, 8), 48880),
    "about_y_60": (8, _about_y(60, 0.84, 1.0), (32, 32, 8), 49104),
    "about_y_1.45": (16, _about_y(5, 1.45, 1.0), (32, 8, 8), 48960),
    "any_8bit": (8, np.array([[425, 67, -181], [-407, 1113, -308], [339, 237, 1088]]) / 1024.0, (32, 8, 16), 49104),
    "any_16bit": (16, np.array([[1360, -373, 335], [17, 657, 16], [-204, 203, 1220]]) / 1024.0, (32, 8, 16), 49104),
}


def _matrix(linear):
    td, th, tw = FRAME
    d, h, w = SRC
    t = np.array([w, h, d]) / 2.0 - linear @ (np.array([tw, th, td]) / 2.0)
    return (np.rint(np.concatenate([linear, t[:, None]], axis=1) * 1024) / 1024).astype(np.float32)


def brick_bytes(linear, tile, bits):
    """The footprint of a tile with its margins, rows an odd number of 16-byte
    units, an odd number of rows per plane."""
    a = 16 // (bits // 8)
    box = [math.ceil(float(sum(abs(linear[i, k]) * (tile[k] - 1) for k in range(3)))) + 5 for i in range(3)]
    units = -(-(box[0] + a - 1) // a)
    return (units | 1) * 16 * (box[1] | 1) * box[2]


def test_bricks_lie_in_the_window():
    for bits, linear, tile, size in MAPS.values():
        assert brick_bytes(_matrix(linear)[:, :3].astype(np.float64), tile, bits) == size
        assert 48 * 1024 - 384 < size <= 48 * 1024


CHILD = """
import sys, numpy as np, torch
from gpu_deconvolution_b200 import api
bits, td, th, tw = (int(a) for a in sys.argv[2:6])
f = np.load(sys.argv[1])
src, m = f["src"], f["m"]
d, h, w = src.shape
pitch = api.source_pitch(bits, w)
dt = torch.int16 if bits == 16 else torch.uint8
t = torch.zeros((d, h, pitch), dtype=dt, device="cuda")
t[..., :w] = torch.from_numpy(src.view(np.int16) if bits == 16 else src).cuda()
out = torch.zeros((td, th, tw), dtype=dt, device="cuda")
api.transform_device(t, pitch, w, h, d, m, tw, th, 0, td, out=out, bits=bits)
torch.cuda.synchronize()
r = out.cpu().numpy()
np.save(sys.argv[1] + ".npy", r.view(np.uint16) if bits == 16 else r)
"""


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(MAPS))
def test_first_call_with_a_brick_near_48k(name, tmp_path):
    bits, linear, _, _ = MAPS[name]
    m = _matrix(linear)
    src = np.random.default_rng(bits).integers(0, 1 << bits, SRC).astype(np.uint16 if bits == 16 else np.uint8)
    path = str(tmp_path / "case.npz")
    np.savez(path, src=src, m=m)
    r = subprocess.run([sys.executable, "-c", CHILD, path, str(bits)] + [str(n) for n in FRAME], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    got = np.load(path + ".npy").astype(np.int64)
    ref = O.transform_volume(src, m.reshape(-1), *FRAME, bits=bits).astype(np.int64)
    diff = np.abs(got - ref)
    assert diff.max() <= 1 and (diff > 0).mean() < 2e-2
