"""The step's reciprocals (rcp2) over the divisors that occur, against CUDA's correctly
rounded ones: a small program compiled from the kernels' own header."""
import subprocess

import pytest

from smectic3d_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include "pencil_kernel.cuh"
using namespace shb;

// C2 = 1 -+ (a rounded value) is 0 or at least 2^-24 (FP64 2^-53) in size; the top is
// where the reciprocal leaves the normal numbers
__global__ void f32(unsigned long long* bad, int lo, int hi) {
  const unsigned long long n = (unsigned long long)(hi - lo + 1) << 23;
  for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < n; i += gridDim.x * 256ull) {
    const float x = __uint_as_float((unsigned(127 + lo + int(i >> 23)) << 23) | unsigned(i & 0x7fffff));
    const float want = __frcp_rn(x);
    const float2 p = rcp2(make_float2(x, -x));
    if (rcp2(x) != want || p.x != want || p.y != -want || rcp2_or_0(x) != want) atomicAdd(bad, 1ull);
  }
}
// |r - 1/x| <= (1/2 + 2^-27) ulp(r): the residual 1 - x r is exact to 2^-53 of itself
__global__ void f64(unsigned long long* bad, int lo, int hi, unsigned long long n) {
  for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < n; i += gridDim.x * 256ull) {
    unsigned long long z = i * 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    z ^= z >> 31;
    if ((i & 0xffff) < 64) z = (i & 1 ? ~0ull : 0ull) << 12 | (i >> 16 & 0xfff);  // ends of the binade
    const unsigned long long e = 1023 + lo + i % (unsigned long long)(hi - lo + 1);
    const double x = __longlong_as_double((long long)(e << 52 | (z & 0xfffffffffffffull)));
    const double r = rcp2(x);
    const double ulp = __longlong_as_double(__double_as_longlong(r) & 0x7ff0000000000000ll) * 0x1p-52;
    if (!(fabs(fma(-x, r, 1.0)) <= x * ulp * (0.5 + 0x1p-27)) || rcp2_or_0(x) != r || rcp2(-x) != -r) atomicAdd(bad, 1ull);
  }
}
__global__ void beyond(int* bad) {
  const float inf = __int_as_float(0x7f800000);
  const double infd = __longlong_as_double(0x7ff0000000000000ll);
  *bad = rcp2_or_0(inf) != 0.0f || rcp2_or_0(-inf) != 0.0f || rcp2_or_0(0x1p126f) != 0.0f || rcp2_or_0(infd) != 0.0 ||
         rcp2_or_0(0x1p1001) != 0.0 || isfinite(rcp2(0.0f)) || isfinite(rcp2(0.0));
}
int main() {
  unsigned long long* bad;
  int* odd;
  if (cudaMallocManaged(&bad, 16) || cudaMallocManaged(&odd, 4)) return 2;
  bad[0] = bad[1] = 0;
  f32<<<1184, 256>>>(bad, -24, 124);
  f64<<<1184, 256>>>(bad + 1, -53, 999, 1ull << 31);
  beyond<<<1, 1>>>(odd);
  if (cudaDeviceSynchronize()) return 3;
  printf("%llu %llu %d\n", bad[0], bad[1], *odd);
  return 0;
}
"""


def test_reciprocals_over_their_range(tmp_path):
    """FP32: equal to __frcp_rn for every significand and exponent; FP64: half an ulp (and
    2^-27 of one, two Newton steps from 20 bits) on 2^31 values.  rcp2_or_0 is 0 beyond."""
    src, exe = tmp_path / "rcp.cu", tmp_path / "rcp"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", f"-I{build.CSRC}",
                    f"-I{build.INCLUDE}", str(src), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0", "0", "0"]
