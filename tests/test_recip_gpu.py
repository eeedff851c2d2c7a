"""The fast modes' reciprocal (recip_mid) against __frcp_rn: every mantissa of every
exponent it is used at, on the device that runs the tests.  Bit equality of
inference with the oracle rests on it."""
import ctypes
import os
import subprocess

import pytest

from tomotopy_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "common.cuh"
__global__ void k_compare(int e0, unsigned long long n, unsigned long long* differ)
{
    unsigned long long d = 0;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const float x = __int_as_float((int)(((unsigned)(e0 + 127) << 23) + (unsigned)i));
        d += __float_as_int(tmtk::recip_mid(x)) != __float_as_int(__frcp_rn(x));
    }
    if (d) atomicAdd(differ, d);
}
// how many of all floats in [2^e0, 2^e1) differ; negative: a CUDA error
extern "C" long long compare(int e0, int e1)
{
    unsigned long long* d = nullptr;
    unsigned long long out = 0;
    cudaError_t e = cudaMalloc(&d, sizeof(out));
    if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof(out));
    if (e == cudaSuccess) {
        k_compare<<<1184, 256>>>(e0, (unsigned long long)(e1 - e0) << 23, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(&out, d, sizeof(out), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? (long long)out : -(long long)e;
}
"""


def test_reciprocal_equals_rounded_division(tmp_path):
    src, so = tmp_path / "recip.cu", tmp_path / "recip.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", build.CSRC,
                    str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(os.fspath(so))
    lib.compare.restype = ctypes.c_longlong
    assert lib.compare(-107, 104) == 0
