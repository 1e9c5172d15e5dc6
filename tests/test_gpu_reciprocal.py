"""The line solves' FP64 reciprocal (hardware seed and one third-order Newton
step) against the IEEE division, over the exponents the pivots can have."""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pllcart3d_b200", "csrc")

SOURCE = r"""
#define PLL_FP64_EXACT 0
#include "line_part.cuh"
__global__ void k(const double* x, double* y, long n)
{
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) y[t] = pll::rcp_<double>(x[t]);
}
extern "C" int rcp_many(const double* x, double* y, long n)
{
    double *dx = nullptr, *dy = nullptr;
    if (cudaMalloc(&dx, 8 * n) != cudaSuccess || cudaMalloc(&dy, 8 * n) != cudaSuccess) return 1;
    cudaMemcpy(dx, x, 8 * n, cudaMemcpyHostToDevice);
    k<<<(unsigned)((n + 255) / 256), 256>>>(dx, dy, n);
    const int bad = cudaMemcpy(y, dy, 8 * n, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(dx);
    cudaFree(dy);
    return bad;
}
"""


def test_reciprocal_within_one_ulp(tmp_path):
    src, lib = tmp_path / "rcp.cu", tmp_path / "librcp.so"
    src.write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I", CSRC, str(src), "-o", str(lib)], check=True)
    L = ctypes.CDLL(str(lib))
    rng = np.random.default_rng(7)
    x = np.concatenate([rng.uniform(1, 2, 1 << 19) * 2.0 ** rng.integers(-300, 300, 1 << 19),
                        1 + np.arange(1 << 18) * 2.0 ** -52, 2 - np.arange(1, 1 << 18) * 2.0 ** -52])
    x = np.ascontiguousarray(x * rng.choice([-1.0, 1.0], x.size))
    y = np.empty_like(x)
    ptr = ctypes.POINTER(ctypes.c_double)
    L.rcp_many.argtypes = [ptr, ptr, ctypes.c_long]
    assert L.rcp_many(x.ctypes.data_as(ptr), y.ctypes.data_as(ptr), x.size) == 0
    # a seed good to 2^-20 leaves 2^-60 after the step, the last fma rounds to
    # half an ulp: no further than one ulp from the correctly rounded quotient
    assert np.all(np.abs(y - 1.0 / x) <= np.spacing(np.abs(1.0 / x)))
