"""A thread's FP32 part of a dot product (Dot, krylov_dev.cuh) (GPU).

A small program with the header is compiled and run: sums of n products for
every n up to the most rows a thread has, positive and of mixed sign, against
the sums in FP64 (exact to 2^-50 here).  Bound: compensated summation leaves
2 u + n u^2 of the sum of magnitudes, u = 2^-24, whatever n is; a plain sum
leaves up to n u, and exceeds the bound among as many trials.
"""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

PROGRAM = r"""
#include <cstdio>
#include <cstdint>
#include "krylov_dev.cuh"
using namespace elfel;

__device__ float number(uint64_t& s, int mixed) {
  s = s * 6364136223846793005ull + 1442695040888963407ull;
  const float v = 1.0f + (float)(s >> 41) * 0x1p-23f;
  return mixed && (s >> 40 & 1) ? -v : v;
}
// worst |sum - exact| / (u sum of magnitudes), in 2^-20: compensated, plain
__global__ void check(int n, int mixed, unsigned long long* res) {
  uint64_t s = (uint64_t)(blockIdx.x * blockDim.x + threadIdx.x) * 7919 + n;
  Dot<float> d;
  Dot<double> e;
  float plain = 0.f;
  double mag = 0.0;
  for (int k = 0; k < n; ++k) {
    const float a = number(s, mixed), b = number(s, 0);
    d.add(a, b);
    e.add((double)a, (double)b);
    plain += a * b;
    mag += fabs((double)a * b);
  }
  atomicMax(res, (unsigned long long)(fabs((double)d.s - e.s) / mag * 0x1p44));
  atomicMax(res + 1, (unsigned long long)(fabs((double)plain - e.s) / mag * 0x1p44));
}

int main() {
  unsigned long long* res;
  if (cudaMallocManaged(&res, 16)) return 2;
  for (int mixed = 0; mixed < 2; ++mixed)
    for (int n = 1; n <= 21; ++n) {
      res[0] = res[1] = 0;
      check<<<512, 256>>>(n, mixed, res);
      if (cudaDeviceSynchronize()) return 2;
      std::printf("%d %d %.6f %.6f\n", mixed, n, res[0] * 0x1p-20, res[1] * 0x1p-20);
    }
  return 0;
}
"""


def test_compensated(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, exe = tmp_path / "dot.cu", tmp_path / "dot"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-O3", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I", os.path.join(ROOT, "elfel.jl_gb300", "csrc"), "-I", os.path.join(ROOT, "include"), str(src),
                    "-o", str(exe)], check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120, check=True).stdout
    rows = [line.split() for line in out.strip().splitlines()]
    assert len(rows) == 42
    for mixed, n, err, plain in rows:
        assert float(err) <= 2.0 + int(n) * 2.0 ** -24, (mixed, n, err)
    assert max(float(r[3]) for r in rows) > 2.1  # the plain sum would not pass
