"""The sines and cosines of sampled angles (csrc/shade.cuh, sincos_f) against
the FP64 functions rounded once, for every float in [-8, 8]: its own range,
[-7, 7], with zeros and denormals, and the FP64 way past it."""
import ctypes
import subprocess

import pytest

from conftest import cuda_available
from yar_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "yar_gpu.h"
#include "shade.cuh"

// out: arguments that differ, one of them
__global__ void compare_kernel(uint32_t first, uint32_t count, unsigned long long* out) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x) {
        const float x = __uint_as_float(first + (uint32_t)i);
        const float2 got = yar::sincos_f(x);
        if (__float_as_uint(got.x) != __float_as_uint((float)sin((double)x)) ||
            __float_as_uint(got.y) != __float_as_uint((float)cos((double)x))) {
            atomicAdd(&out[0], 1ull);
            out[1] = first + (uint32_t)i;
        }
    }
}
extern "C" int compare(uint32_t first, uint32_t count, unsigned long long* out) {
    unsigned long long* d = nullptr;
    cudaError_t e = cudaMalloc(&d, 16);
    if (e == cudaSuccess) e = cudaMemset(d, 0, 16);
    if (e == cudaSuccess) compare_kernel<<<152 * 16, 128>>>(first, count, d);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(out, d, 16, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
"""


@pytest.fixture(scope="module")
def compare(tmp_path_factory):
    if not cuda_available():
        pytest.skip("no CUDA device")
    d = tmp_path_factory.mktemp("sincos")
    (d / "sincos.cu").write_text(SOURCE)
    subprocess.run([build._nvcc()] + build.GENCODE + build.NVCC_FLAGS +
                   ["-shared", str(d / "sincos.cu"), "-o", str(d / "sincos.so")], check=True)
    f = ctypes.CDLL(str(d / "sincos.so")).compare
    f.argtypes = [ctypes.c_uint32, ctypes.c_uint32, ctypes.POINTER(ctypes.c_ulonglong)]
    return f


@pytest.mark.parametrize("sign", [0, 0x80000000])
def test_every_float(compare, sign):
    out = (ctypes.c_ulonglong * 2)()
    assert compare(sign, 0x41000001, out) == 0  # 8.0 is 0x41000000
    assert out[0] == 0, "%d differ, 0x%08x for one" % (out[0], out[1])
