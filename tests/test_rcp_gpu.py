"""The reciprocal of a softmax sum in the soft scans (rcp_normal of csrc/slotscan_common.cuh) against the division."""
import ctypes
import math
import os
import shutil
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include "slotscan_common.cuh"
__global__ void rcp_kernel(const double* x, double* y, long long n) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i < n) y[i] = slotscan::rcp_normal(x[i]);
}
extern "C" int rcp(const double* x, double* y, long long n) {
    rcp_kernel<<<(unsigned)((n + 255) / 256), 256>>>(x, y, n);
    return (int)cudaDeviceSynchronize();
}
"""


def test_rcp_normal_against_the_division(tmp_path):
    """Sums from exp(-600) to 256 exp(600), random mantissas and those at the ends of a binade: never more than one unit in the
    last place from 1 / s (its own rounding is half a unit, the iteration's remainder below 2^-4 of one)."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, so = tmp_path / "rcp.cu", tmp_path / "librcp.so"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC",
                    "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "smal-memory-llm_b200", "csrc"),
                    str(src), "-o", str(so), "-lcudart"], check=True)
    fn = ctypes.CDLL(str(so)).rcp
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong]
    gen = torch.Generator(device="cuda").manual_seed(1)
    u = torch.rand(1 << 22, device="cuda", dtype=torch.float64, generator=gen)
    x = torch.exp((600 + math.log(256)) * u - 600 * (1 - u))
    near = torch.arange(-64, 64, device="cuda")                # bit patterns around every power of two of the range
    powers = torch.ldexp(torch.ones(1730, device="cuda", dtype=torch.float64), torch.arange(-865, 865, device="cuda"))
    x = torch.cat([x, (powers.view(torch.int64)[:, None] + near).view(torch.float64).flatten()])
    y = torch.empty_like(x)
    assert fn(x.data_ptr(), y.data_ptr(), x.numel()) == 0
    assert ((y.view(torch.int64) - (1.0 / x).view(torch.int64)).abs() <= 1).all()
