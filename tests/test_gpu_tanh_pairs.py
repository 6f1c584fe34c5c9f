"""The packed tanh of the plain network against the scalar one it restates: the same bits for every FP32 input in
either half of a pair (the halves of a pair hold unrelated values), NaN for NaN.

The plain network's outputs are compared bit for bit with the CPU restatement elsewhere, at the pre-activations of a few
thousand separations; the packed form's reciprocal (one Newton step) is equal to the scalar division only if it is so
for every input, so every input is tried.
"""
import ctypes
import subprocess

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from hignn_b200 import build as B  # noqa: E402

SOURCE = r"""
#include <cstdint>
#include "tanh_f32.cuh"
#include "tanh_f32x2.cuh"

__device__ bool same(float a, float b) { return a != a ? b != b : __float_as_uint(a) == __float_as_uint(b); }

// every 32-bit pattern i in the low half, the odd multiple of it (a permutation of the patterns) in the high half
__global__ void k_compare(unsigned long long* bad, uint32_t* first) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 32);
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t lo = (uint32_t)i, hi = lo * 2654435761u;
    const float x = __uint_as_float(lo), y = __uint_as_float(hi);
    const hignn::f2 t = hignn::tanh_f32x2(hignn::f2_make(x, y));
    if (!same(hignn::tanh_f32(x), hignn::f2_lo(t)) && atomicAdd(bad, 1ull) == 0) *first = lo;
    if (!same(hignn::tanh_f32(y), hignn::f2_hi(t)) && atomicAdd(bad, 1ull) == 0) *first = hi;
  }
}

extern "C" int compare(unsigned long long* bad, unsigned* first) {
  void* d = nullptr;
  if (cudaMalloc(&d, 16) != cudaSuccess) return 1;
  cudaMemset(d, 0, 16);
  k_compare<<<148 * 8, 256>>>((unsigned long long*)d, (uint32_t*)d + 2);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(bad, d, 8, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(first, (char*)d + 8, 4, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
"""


def test_every_input(tmp_path):
    src, lib = tmp_path / "pairs.cu", tmp_path / "pairs.so"
    src.write_text(SOURCE)
    subprocess.run([B.NVCC, "-std=c++17", "-O3", *B.ARCH, "-I", B.CSRC, "-shared", "-Xcompiler", "-fPIC", "-cudart",
                    "static", "-o", str(lib), str(src)], check=True)
    bad, first = ctypes.c_ulonglong(), ctypes.c_uint()
    assert ctypes.CDLL(str(lib)).compare(ctypes.byref(bad), ctypes.byref(first)) == 0
    assert bad.value == 0, f"{bad.value} inputs differ, {first.value:#010x} among the first"
