"""fast_rcp and fast_div (fastdiv64.cuh) against the device's IEEE division (GPU).

A small program with the header is compiled and run.  Bounds, from the header:
with y exact to 2^-40 after the first step, the second leaves 1 / x to 2^-80
before its last rounding, so the result is the rounded quotient or its
neighbour; the same for a quotient corrected by its remainder.  Arguments: random
significands over all exponents and around the two exponents where the forms
change, both signs; zeros, subnormals, infinities and NaN give what the division
gives.
"""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "elfel.jl_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdint>
#include "fastdiv64.cuh"
using namespace elfel;

__device__ uint64_t mix(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__device__ double number(uint64_t h, int e) {  // significand and sign from h, biased exponent e
  return __longlong_as_double((long long)((h & 0x800fffffffffffffull) | ((uint64_t)e << 52)));
}
__device__ bool special(double v) {  // not a normal number
  const int e = (int)((__double_as_longlong(v) >> 52) & 0x7ff);
  return e == 0 || e == 2047;
}
// distance in units in the last place; not comparable: -1
__device__ long long ulps(double got, double want) {
  const long long g = __double_as_longlong(got), w = __double_as_longlong(want);
  if (g == w || (isnan(got) && isnan(want))) return 0;
  if (isnan(got) || isnan(want) || (g ^ w) < 0) return -1;
  return g > w ? g - w : w - g;
}
// res: worst fast_rcp, worst fast_div, wrong specials, compared
__global__ void check(int n, long long* res) {
  const int stride = gridDim.x * blockDim.x;
  long long wr = 0, wd = 0, bad = 0, cnt = 0;
  const int edges[8] = {58, 59, 60, 61, 1979, 1980, 1981, 1982};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint64_t h = mix(2 * (uint64_t)i + 1), k = mix(2 * (uint64_t)i + 2);
    const double x = number(h, i & 1 ? edges[(i >> 1) & 7] : 1 + (int)(mix(k) % 2046));
    const double a = number(k, 1 + (int)(mix(h) % 2046));
    const double y = fast_rcp(x), r = 1.0 / x, q = fast_div(a, x), d = a / x;
    const long long u = ulps(y, r), v = ulps(q, d);
    if (special(r)) bad += u != 0;  // through the division
    else if (u < 0) ++bad;
    else wr = max(wr, u);
    if (special(d)) {
      bad += v != 0;  // through the division
    } else if (v < 0) {
      ++bad;
    } else {
      wd = max(wd, v);
    }
    cnt += 2;
  }
  atomicMax(res, wr);
  atomicMax(res + 1, wd);
  atomicAdd((unsigned long long*)(res + 2), (unsigned long long)bad);
  atomicAdd((unsigned long long*)(res + 3), (unsigned long long)cnt);
}
__global__ void specials(long long* res) {
  const double inf = __longlong_as_double(0x7ff0000000000000LL), nan = __longlong_as_double(0x7ff8000000000000LL);
  const double v[] = {0.0, -0.0, inf, -inf, nan, 0x1p-1074, -0x1p-1074, 0x1p-1023, 0x1.fffffffffffffp-1023, 0x1p-1022,
                      1.0, -3.0, 0x1p1023, 0x1.fffffffffffffp1023, -0x1.fffffffffffffp1023, 0x1p-963, 0x1p957};
  const int n = sizeof(v) / sizeof(v[0]);
  long long bad = 0;
  for (int i = 0; i < n; ++i) {
    const double y = fast_rcp(v[i]);
    if (ulps(y, 1.0 / v[i]) != 0) ++bad;
    for (int j = 0; j < n; ++j) {
      const double q = fast_div(v[j], v[i]), d = v[j] / v[i];
      const long long u = ulps(q, d);
      if (!(u == 0 || (!special(d) && u == 1))) ++bad;
    }
  }
  res[4] = bad;
}

int main() {
  long long *res, h[5];
  if (cudaMallocManaged(&res, sizeof(h))) return 2;
  for (int k = 0; k < 5; ++k) res[k] = 0;
  check<<<304, 256>>>(1 << 24, res);
  specials<<<1, 1>>>(res);
  if (cudaDeviceSynchronize()) return 2;
  for (int k = 0; k < 5; ++k) h[k] = res[k];
  std::printf("%lld %lld %lld %lld %lld\n", h[0], h[1], h[2], h[3], h[4]);
  return 0;
}
"""


def test_against_the_division(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, exe = tmp_path / "fastdiv.cu", tmp_path / "fastdiv"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", "-I", CSRC, str(src), "-o",
                    str(exe)], check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120, check=True)
    rcp, div, wrong, compared, specials = map(int, out.stdout.split())
    assert compared == 2 << 24
    assert rcp <= 1 and div <= 1 and wrong == 0 and specials == 0, out.stdout
