"""Opt-in of a kernel to large shared memory, which the CUDA runtime keeps per
device: a process that uses a second device opts in there too, once, and a
refused opt-in is tried again.  The host code runs against a stand-in for the
runtime; the convolution GEMMs' configure() is taken from its source."""
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "gpu_deconvolution_b200", "csrc")

RUNTIME = """
#pragma once
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize };
enum cudaDeviceAttr { cudaDevAttrMultiProcessorCount };
extern int device, calls, refuse;
inline cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
inline cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int d) { *v = 100 + d; return cudaSuccess; }
template <typename K>
cudaError_t cudaFuncSetAttribute(K, cudaFuncAttribute, int)
{
    calls++;
    return refuse ? cudaErrorInvalidValue : cudaSuccess;
}
"""

MAIN = """
#include <atomic>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#define FMVD_CHECK(call) ((call) == cudaSuccess)
%s
int device = 0, calls = 0, refuse = 1;
void kernel() {}
int main()
{
    %s
    const bool refused = !go();
    refuse = 0;
    bool ok = go() && go();
    printf("%%d %%d %%d ", refused, ok, calls);
    device = 1;
    ok = go() && go();
    device = 0;
    ok = ok && go();
    printf("%%d %%d\\n", ok, calls);
}
"""


def _run(tmp_path, helpers, go):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(MAIN % (helpers, go))
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-I" + str(tmp_path), "-I" + CSRC, str(tmp_path / "main.cpp"), "-o", exe],
                   check=True)
    return subprocess.run([exe], capture_output=True, text=True, check=True, timeout=60).stdout.split()


def test_allow_smem(tmp_path):
    got = _run(tmp_path, '#include "smem_opt_in.h"', """
    std::atomic<unsigned long long> devices{0};
    const auto go = [&]() { return fmvd::allow_smem(kernel, 60000, devices) == cudaSuccess; };""")
    assert got == ["1", "1", "2", "1", "3"]


def test_convolution_configure(tmp_path):
    text = open(os.path.join(CSRC, "unet_gemm.cu")).read()
    body = re.search(r"^template <typename K>\nbool configure\(.*?^}\n", text, re.M | re.S).group(0)
    got = _run(tmp_path, '#include "smem_opt_in.h"\nusing namespace fmvd;\n' + body, """
    std::atomic<unsigned long long> devices{0};
    const auto go = [&]() { int sms = 0; return configure(kernel, 60000, devices, sms) && sms == 100 + device; };""")
    assert got == ["1", "1", "2", "1", "3"]
