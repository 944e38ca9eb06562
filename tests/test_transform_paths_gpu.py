"""The resampler's two kernels on maps that both can take: a map that turns the
volume about the y axis (the row-walking kernel) and the same map with a
coupling far below rounding (the general kernel) sample the same coordinates,
so samples and float values are equal bit for bit, whatever the frame's
remainders, the step along y, the part of the volume seen, and the output.
The coefficients are multiples of 2^-9, so that every product and sum is exact:
a coordinate that had to be rounded could lie half way between two floats, and
there the tiny coupling would decide the rounding."""
import numpy as np
import pytest

from gpu_deconvolution_b200 import api


def _map(angle, sy, ty, zs, centre, shift):
    c, s = np.cos(np.deg2rad(angle)), np.sin(np.deg2rad(angle))
    m = np.array([[c, 0, s, 0], [0, sy, 0, ty], [-s / zs, 0, c / zs, 0]])
    m[0, 3] = centre[0] - c * centre[2] - s * centre[3] + shift
    m[2, 3] = centre[1] - (-s * centre[2] + c * centre[3]) / zs + shift / 3
    return (np.rint(m * 512) / 512).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [16, 8])
@pytest.mark.parametrize("frame", [(11, 37, 45), (8, 32, 32), (1, 1, 1), (17, 67, 70)])
@pytest.mark.parametrize("angle,sy,ty,zs", [(0, 1, 0.25, 1), (90, 1, -3.5, 3), (37, 1, 40, 2), (180, 0.5, 1, 1.5),
                                            (270, 1.7, -2, 2), (20, -1, 45.5, 1), (65, 0, 7.125, 2), (10, 9, 0, 1)])
def test_row_walk_equals_general(bits, frame, angle, sy, ty, zs):
    import torch
    td, th, tw = frame
    d, h, w = 19, 50, 61
    g = torch.Generator(device="cuda").manual_seed(bits + td)
    pitch = api.source_pitch(bits, w)
    src = torch.zeros((d, h, pitch), dtype=torch.int16 if bits == 16 else torch.uint8, device="cuda")
    src[..., :w] = torch.randint(-(1 << 15) if bits == 16 else 0, 1 << (15 if bits == 16 else 8), (d, h, w),
                                 generator=g, device="cuda").to(src.dtype)
    src[3:6, 10:20, 10:20] = -1 if bits == 16 else 255  # saturated samples
    m = _map(angle, sy, ty, zs, (w / 2, d / 2, tw / 2, td / 2), 0.3)
    tiny = m.copy()
    tiny[0, 1] = tiny[1, 0] = 1e-32  # no longer a turn about y; adds nothing to any coordinate
    assert np.array_equal(m[0, 1:2], [0]) and tiny[0, 1] > 0
    for z0, nz in ((0, td), (td // 2, td - td // 2)):
        res = []
        for mat in (m, tiny):
            for with_s, with_f in ((True, True), (True, False), (False, True)):
                out = torch.zeros((nz, th, tw), dtype=src.dtype, device="cuda") if with_s else None
                outf = torch.zeros((nz, th, tw), dtype=torch.float32, device="cuda") if with_f else None
                api.transform_device(src, pitch, w, h, d, mat, tw, th, z0, nz, out=out, out_f32=outf, bits=bits)
                res.append((out, outf))
        torch.cuda.synchronize()
        samples = [r[0] for r in res if r[0] is not None]
        floats = [r[1] for r in res if r[1] is not None]
        assert all(torch.equal(samples[0], s) for s in samples[1:])
        assert all(torch.equal(floats[0], f) for f in floats[1:])
