"""The convolution GEMMs' warps stay together when a wait gives up: a warp's
lanes poll and read the failure flag each for themselves, but the operations
that follow (elect.sync of an MMA or a commit, tensor-memory loads) wait for
all 32 of them, so the lanes must leave a loop together.  Runs the kernels'
device code on the CPU with stand-ins for the hardware (unet_roles/emulator.cpp):
waits that time out for some lanes of a role end with the status set, and none
leaves a lane behind."""
import os
import re
import subprocess

import pytest

from conftest import ROOT

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(ROOT, "gpu_deconvolution_b200", "csrc")
ALL, SOME = 0xFFFFFFFF, 0x00F0FF31
MMA = {"persistent": 5, "halo": 5, "wgrad": 1}
PRODUCER = {"persistent": 4, "halo": 4, "wgrad": 0}
OTHER = {"persistent": 2, "halo": 2, "wgrad": 3}  # an epilogue warp; a warp of the bias sums


@pytest.fixture(scope="module")
def emulator(tmp_path_factory):
    out = tmp_path_factory.mktemp("roles")
    text = open(os.path.join(CSRC, "unet_gemm.cu")).read()
    device = text[:re.search(r"^// -+ host$", text, re.M).start()]
    device = re.sub(r"^#include.*$", "", device, flags=re.M)
    device = device.replace("extern __shared__ uint8_t smem_raw[];", "uint8_t *const smem_raw = smem_block;")
    device = re.sub(r"__launch_bounds__\([^)]*\)", "", device.replace("__shared__", "static"))
    (out / "device.inc").write_text(device + "\n} }\n")
    exe = str(out / "emulator")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-pthread", "-I" + str(out), "-I" + CSRC, "-I/usr/local/cuda/include",
                    os.path.join(HERE, "unet_roles", "emulator.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("kernel", ["persistent", "halo", "wgrad"])
@pytest.mark.parametrize("role,lanes,call", [("none", 0, -1), ("mma", SOME, 0), ("mma", SOME, 5), ("mma", ALL, 3),
                                             ("other", SOME, 2), ("producer", 1, 0), ("producer", 1, 1),
                                             ("producer", 1, 2)])
def test_lanes_leave_together(emulator, kernel, role, lanes, call):
    warp = {"none": 0, "mma": MMA, "other": OTHER, "producer": PRODUCER}[role]
    warp = warp if isinstance(warp, int) else warp[kernel]
    seeds = 3
    r = subprocess.run([emulator, kernel, str(warp), hex(lanes), str(call), str(seeds)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
    assert int(r.stdout) == (0 if role == "none" else seeds)
