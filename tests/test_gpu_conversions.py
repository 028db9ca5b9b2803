"""The integer forms of the FP32 <-> FP64 conversions (csrc/tc_ptx.cuh) and the short reciprocals
(csrc/recip.cuh) against the conversions, divisions and square roots they stand for.

Conversions: the same bits for every input.  Reciprocals: a seed of 2^-21 and a cubic step leave
2^-63, the last additions round by half an ulp and what goes into them by a quarter at most: within
one ulp (two against 1 / sqrt, which rounds twice)."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "mpskit.jl_gb300", "csrc")

PROGRAM = r"""
#include "recip.cuh"
#include <cstdio>
using namespace gb;

__device__ unsigned long long mix(unsigned long long x) {
  x ^= x >> 33; x *= 0xff51afd7ed558ccdull; x ^= x >> 29; x *= 0xc4ceb9fe1a85ec53ull;
  return x ^ (x >> 32);
}
__device__ bool same(float a, float b) {
  return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}
__device__ bool same(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b);
}
__device__ void check_double(double x, int* bad) {
  if (!same(to_float(x), (float)x)) atomicAdd(&bad[0], 1);
}
__device__ void check_float(float x, int* bad) {
  if (!same(to_double(x), (double)x)) atomicAdd(&bad[1], 1);
}
// distance in units of the last place of the correctly rounded value
__device__ long long ulps(double a, double b) {
  return llabs(__double_as_longlong(a) - __double_as_longlong(b));
}
__global__ void run(int* bad) {
  const unsigned long long n = 1ull << 24;
  for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < n; i += gridDim.x * 256ull) {
    // every FP32 pattern with 16 of its lower bits, all exponents
    check_float(__uint_as_float((unsigned)(i << 8) | (unsigned)(mix(i) & 0xff)), bad);
    const unsigned long long r = mix(i);
    check_double(__longlong_as_double((long long)r), bad);  // all exponents of FP64
    // around every FP32 value: exact, the tie above it, and its neighbours
    const double f = (double)__uint_as_float((unsigned)(r >> 32));
    const long long u = __double_as_longlong(f);
    for (long long tie = 0; tie < 2; ++tie)
      for (long long k = -1; k <= 1; ++k)
        check_double(__longlong_as_double(u + (tie << 28) + k), bad);
    // the ends of FP32's normal range and its subnormals
    const double s = __hiloint2double((int)(0x36800000u + (unsigned)(r % 0x02000000u)),
                                      (int)(r >> 32));
    check_double(s, bad);
    check_double(-s, bad);
    const double l = __hiloint2double((int)(0x47e00000u + (unsigned)(r % 0x00300000u)),
                                      (int)(r >> 32));
    check_double(l, bad);
    // reciprocals: exponents -1000 to 1000, any mantissa, and mantissas next to 1 and 2
    const int e = (int)(r % 2001u) + 23;
    unsigned long long m = mix(r) >> 12;
    if (i % 8 == 0) m &= 0xff;
    if (i % 8 == 1) m |= 0xfffffffffff00ull;
    const double d = __longlong_as_double((long long)(((unsigned long long)e << 52) | m));
    if (ulps(inverse(d), 1.0 / d) > 1) atomicAdd(&bad[2], 1);
    if (ulps(inv_sqrt(d), rsqrt(d)) > 2 || ulps(inv_sqrt(d), 1.0 / sqrt(d)) > 2)
      atomicAdd(&bad[3], 1);
  }
}
int main() {
  int *bad, h[4];
  if (cudaMalloc(&bad, sizeof(h)) != cudaSuccess) return 2;
  cudaMemset(bad, 0, sizeof(h));
  run<<<608, 256>>>(bad);
  if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
  std::printf("%d %d %d %d\n", h[0], h[1], h[2], h[3]);
}
"""


def test_conversions_and_reciprocals(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, exe = tmp_path / "conv.cu", tmp_path / "conv"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2",
                    "--expt-relaxed-constexpr", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0
    assert out.stdout.split() == ["0"] * 4
