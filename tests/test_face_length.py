"""Length of the face vector and its reciprocal (physics.cuh), over every FP32
mantissa: their product is 1 within the error of one reciprocal (2^-23) and
half the rounding of the comparison, 1.5 x 2^-23 in all; a reciprocal root used
for both leaves twice its error there."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cmath>
#include "cc_common.h"
#include "physics.cuh"
__global__ void k_worst(unsigned *worst) {
  const unsigned n = 1u << 24, step = gridDim.x * blockDim.x;  // [1, 4): every mantissa at both parities of the exponent
  float w = 0.0f;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
    float len, inv;
    ccb::length_and_reciprocal(__uint_as_float(0x3f800000u + i), len, inv);
    w = fmaxf(w, (float)fabs((double)len * (double)inv - 1.0));
  }
  atomicMax(worst, __float_as_uint(w));
}
int main() {
  unsigned *d = nullptr, bits = 0;
  if (cudaMalloc(&d, sizeof bits) != cudaSuccess || cudaMemset(d, 0, sizeof bits) != cudaSuccess) return 1;
  k_worst<<<296, 256>>>(d);
  if (cudaMemcpy(&bits, d, sizeof bits, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  cudaFree(d);
  float w;
  static_assert(sizeof w == sizeof bits, "");
  __builtin_memcpy(&w, &bits, sizeof w);
  std::printf("%.9g\n", w);
  return 0;
}
"""


@pytest.mark.gpu
def test_product_of_length_and_reciprocal(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, exe = tmp_path / "length.cu", tmp_path / "length"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(ROOT, "combustioncodegpu_b200", "csrc"), "-o", str(exe), str(src)], check=True,
                   timeout=300)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    assert 0.0 < float(out) <= 1.5 * 2.0 ** -23
