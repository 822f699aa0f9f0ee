"""The device's sRGB8 quantisation against the exact thresholds, over every
float from 0 to 1 and the values outside: a kernel compiled from the engine's
own header counts the values whose code is not the number of thresholds that
they have reached."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r'''
#include "oit_device.cuh"

// Every float in [first, first + count) as bits: its code against a search of the thresholds.
__global__ void check(uint32_t first, uint32_t count, const float* thr, unsigned long long* wrong) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < count; i += gridDim.x * (uint64_t)blockDim.x) {
    const float c = __uint_as_float(first + (uint32_t)i);
    uint32_t lo = 0, hi = 255;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) / 2;
      if (c >= thr[mid]) lo = mid + 1; else hi = mid;
    }
    if (oitd::srgb_encode(c) != lo) atomicAdd(wrong, 1ull);
  }
}

extern "C" long long mismatches(uint32_t first, uint32_t count, const float* thr_host) {
  float* thr = nullptr;
  unsigned long long* wrong = nullptr;
  unsigned long long n = 0;
  if (cudaMalloc(&thr, 1024) != cudaSuccess || cudaMalloc(&wrong, 8) != cudaSuccess) return -1;
  cudaMemcpy(thr, thr_host, 1024, cudaMemcpyHostToDevice);
  cudaMemset(wrong, 0, 8);
  check<<<1216, 256>>>(first, count, thr, wrong);
  const cudaError_t e = cudaMemcpy(&n, wrong, 8, cudaMemcpyDeviceToHost);
  cudaFree(thr);
  cudaFree(wrong);
  return e == cudaSuccess ? (long long)n : -1;
}
'''


@pytest.fixture(scope='module')
def checker(engine, tmp_path_factory):
    from vk_order_independent_transparency_gb300 import _build
    d = tmp_path_factory.mktemp('srgb')
    src, lib = os.path.join(d, 'check.cu'), os.path.join(d, 'check.so')
    with open(src, 'w') as f:
        f.write(SOURCE)
    subprocess.run([_build.nvcc(), *_build.ARCH, '-O3', '-std=c++17', '-shared', '-Xcompiler', '-fPIC', '-I',
                    _build.CSRC, src, '-o', lib], check=True, capture_output=True)
    so = ctypes.CDLL(lib)
    so.mismatches.restype = ctypes.c_longlong
    so.mismatches.argtypes = [ctypes.c_uint32, ctypes.c_uint32, ctypes.c_void_p]
    thr = np.ascontiguousarray(engine.srgb_tables()[0])
    return lambda first, count: so.mismatches(first, count, thr.ctypes.data)


@pytest.mark.parametrize('first,count', [
    (0x00000000, 0x3F800001),  # 0 .. 1
    (0x3F800000, 0x00100000),  # 1 and above
    (0x7F7FFF00, 0x00800100),  # the largest floats, infinity, every positive NaN (which reaches no threshold)
    (0x80000000, 0x7F800001),  # -0 .. -infinity
])
def test_every_float(checker, first, count):
    assert checker(first, count) == 0
