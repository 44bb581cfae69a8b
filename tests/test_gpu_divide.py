"""mkpp::divide and mkpp::max_abs (csrc/mkpp_device.cuh) against the hardware's
division and fmax, bit for bit, on the GPU: random operands over all bit
patterns and over the normal range, significands at the ends of their range,
numerators close to the denominator, quotients next to a rounding midpoint,
reciprocals, and every pair of special values."""

import ctypes as C
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parent.parent / "mkpp_gb300" / "csrc"

SOURCE = r"""
#include "mkpp_device.cuh"
typedef unsigned long long u64;
__device__ u64 mix(u64 x) {
  x ^= x >> 30; x *= 0xbf58476d1ce4e5b9ull; x ^= x >> 27; x *= 0x94d049bb133111ebull; return x ^ (x >> 31);
}
__device__ bool same(double x, double y) {
  return __double_as_longlong(x) == __double_as_longlong(y) || (x != x && y != y);
}
__device__ void check(double a, double b, u64* bad) {
  if (!same(mkpp::divide(a, b), __ddiv_rn(a, b))) atomicAdd(bad, 1ull);
  if (!same(mkpp::max_abs(a, b), fmax(fabs(a), fabs(b)))) atomicAdd(bad + 1, 1ull);
}
__global__ void run(u64* bad, int rounds) {
  const u64 t = blockIdx.x * (u64)blockDim.x + threadIdx.x;
  const u64 M = (1ull << 52) - 1;
  for (int i = 0; i < rounds; ++i) {
    const u64 x = mix(2 * (t * rounds + i) + 1), y = mix(x + 0x9e3779b97f4a7c15ull);
    u64 ma = x & M, mb = y & M;
    switch (i & 7) {
      case 1: mb = M - (y & 0xff); break;
      case 2: mb = y & 0xff; break;
      case 3: ma = x & 0xff; mb = M - (y & 0xffffff); break;
      case 4: ma = 0; break;
      case 5: mb = (mb & ~((1ull << 22) - 1)) | ((1ull << 22) - 1 - (x >> 60)); break;
      case 6: ma = (mb + ((x >> 50) & 7) - 3) & M; break;
      case 7: {
        const double q = __longlong_as_double((1023ull << 52) | ma), b = __longlong_as_double((1023ull << 52) | mb);
        ma = (u64)__double_as_longlong(q * b * (1.0 + 1.1102230246251565e-16)) & M;
        break;
      }
    }
    const u64 ea = 1 + (x >> 53) % 2046, eb = 1 + (y >> 53) % 2046, s = 1ull << 63;
    check(__longlong_as_double((ea << 52) | ma | (x & s)), __longlong_as_double((eb << 52) | mb | (y & s)), bad);
    check(__longlong_as_double((long long)x), __longlong_as_double((long long)y), bad);
    check(1.0, __longlong_as_double((eb << 52) | mb | (y & s)), bad);
  }
  if (t == 0) {
    const u64 sp[] = {0, 1, M, M + 1, M + 2, 0x3ff0000000000000ull, 0x3fefffffffffffffull, 0x4008000000000000ull,
                      0x0020000000000001ull, 0x7fe0000000000000ull, 0x7fefffffffffffffull, 0x7ff0000000000000ull,
                      0x7ff8000000000000ull, 0x3cb0000000000001ull, 0x4330000000000001ull};
    for (u64 a : sp)
      for (u64 b : sp)
        for (int k = 0; k < 4; ++k)
          check(__longlong_as_double((long long)(a | ((u64)(k & 1) << 63))),
                __longlong_as_double((long long)(b | ((u64)(k >> 1) << 63))), bad);
  }
}
extern "C" int divide_check(unsigned long long* out) {
  u64* bad;
  if (cudaMalloc(&bad, 16) != cudaSuccess) return 1;
  cudaMemset(bad, 0, 16);
  run<<<608, 256>>>(bad, 512);
  const int rc = (int)cudaMemcpy(out, bad, 16, cudaMemcpyDeviceToHost);
  cudaFree(bad);
  return rc;
}
"""


def test_divide_is_the_correctly_rounded_division(tmp_path):
    from mkpp_gb300 import build

    (tmp_path / "divide.cu").write_text(SOURCE)
    so = tmp_path / "divide.so"
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false", "-shared", "-Xcompiler", "-fPIC",
                    f"-I{CSRC}", str(tmp_path / "divide.cu"), "-o", str(so)], check=True)
    bad = (C.c_ulonglong * 2)()
    assert C.CDLL(str(so)).divide_check(bad) == 0
    assert list(bad) == [0, 0]
