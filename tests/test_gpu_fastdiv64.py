"""fast_rcp, fast_div and times_rcp (fastdiv64.cuh) against the device's IEEE division (GPU).

A small program with the header is compiled and run.  Bounds, from the header:
with y exact to 2^-40 after the first step, the second leaves 1 / x to 2^-80
before its last rounding, so the result is the rounded quotient or its
neighbour; the same for a quotient corrected by its remainder, one more rounding
without the correction.  Arguments: random
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
// res: worst fast_rcp, worst fast_div, wrong specials, compared, (specials), worst times_rcp
__global__ void check(int n, long long* res) {
  const int stride = gridDim.x * blockDim.x;
  long long wr = 0, wd = 0, wt = 0, bad = 0, cnt = 0;
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
    const double t = times_rcp(a, x, newton_rcp(x));
    const long long w = ulps(t, d);
    const int ex = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
    if (ex < 60 || ex > 1980) bad += w != 0;  // the division
    else if (!special(d) && !special(t)) wt = max(wt, w < 0 ? 1000 : w);
    cnt += 2;
  }
  atomicMax(res, wr);
  atomicMax(res + 1, wd);
  atomicAdd((unsigned long long*)(res + 2), (unsigned long long)bad);
  atomicAdd((unsigned long long*)(res + 3), (unsigned long long)cnt);
  atomicMax(res + 5, wt);
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
  long long *res, h[6];
  if (cudaMallocManaged(&res, sizeof(h))) return 2;
  for (int k = 0; k < 6; ++k) res[k] = 0;
  check<<<304, 256>>>(1 << 24, res);
  specials<<<1, 1>>>(res);
  if (cudaDeviceSynchronize()) return 2;
  for (int k = 0; k < 6; ++k) h[k] = res[k];
  std::printf("%lld %lld %lld %lld %lld %lld\n", h[0], h[1], h[2], h[3], h[4], h[5]);
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
    rcp, div, wrong, compared, specials, times = map(int, out.stdout.split())
    assert compared == 2 << 24
    assert rcp <= 1 and div <= 1 and times <= 2 and wrong == 0 and specials == 0, out.stdout


@pytest.mark.parametrize("method", ["pcg64", "batch"])
@pytest.mark.parametrize("scale", [1.0, 1e-150, 1e-160, 1e140])
def test_scalars_near_the_ends_of_the_range(E, gpu, method, scale):
    """A right-hand side of 1e-160, whose dot products are subnormal: the steps divide by them.  Two
    unknowns with condition number 7 / 3: a residual of 1e-9 leaves 3e-9; subnormal sums of 1e-320 have 11 bits,
    so with them the answer is asked to 1 %."""
    import numpy as np
    import scipy.sparse as sp

    A = sp.csr_matrix(np.array([[2.5, -1.0], [-1.0, 2.5]]))
    F = scale * np.array([0.3, -1.1])
    c = A.tocoo()
    a = E.start(E.SysmatAssemblerSparse(0.0), 2, 2)
    a._chunks.append((c.row.astype(np.int64) + 1, c.col.astype(np.int64) + 1, c.data.astype(np.float64)))
    E.finish(a)
    T = np.zeros(2)
    if method == "batch":
        b = E.BatchSolver("pcg64", capacity=1)
        s = b.add(a, T, 2, F=F, rtol=1e-9)
        T, st = b.run()[s]
        b.close()
    else:
        st = E.solve(T, a, F, 2, method=method, rtol=1e-9)
    want = np.linalg.solve(A.toarray(), F / scale)
    assert st["converged"] and np.abs(T / scale - want).max() <= (0.01 if scale < 1e-155 else 3e-9)
