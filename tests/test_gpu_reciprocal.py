"""The reciprocal of the lattice sums' elimination steps (csrc/reciprocal.cuh) against
the division. An approximation r0 with |1 - d r0| <= 2^-20 and two Newton-Raphson steps
leave 2^-80 before the last rounding, so that the result is within half a unit in the
last place of 1 / d but for the rounding of the residual (2^-93): at most one from the
correctly rounded quotient. Outside (1e-290, 1e290) it is the quotient. Exponents over
the whole range, mantissas next to 1 and 2, both range limits and their neighbours,
zeros, subnormals, infinities, NaN. Compiled here."""
import os
import shutil
import subprocess

import pytest

from pyqcm_b200 import build

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>
#include "reciprocal.cuh"
__global__ void k(int n, const double *d, double *r, double *q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    r[i] = qed::reciprocal(d[i]);
    q[i] = 1.0 / d[i];
  }
}
int main() {
  std::vector<double> h;
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> m(1.0, 2.0);
  for (int e = -1074; e <= 1023; ++e) {
    for (int i = 0; i < 500; ++i) h.push_back(std::ldexp(m(g), e));
    for (double x : {1.0, std::nextafter(1.0, 2.0), std::nextafter(2.0, 1.0), 1.5, std::nextafter(1.0, 0.0)})
      h.push_back(std::ldexp(x, e));
  }
  for (double x : {1e-290, 1e290})
    for (double y : {x, std::nextafter(x, 0.0), std::nextafter(x, 1e300), 0.5 * x, 2.0 * x}) h.push_back(y);
  const size_t whole = h.size();
  for (size_t i = 0; i < whole; i += 97) h.push_back(-h[i]);
  const double inf = std::numeric_limits<double>::infinity();
  for (double x : {0.0, -0.0, inf, -inf, std::nan(""), 4.9e-324, 2.2250738585072014e-308}) h.push_back(x);
  const int n = (int)h.size();
  double *d, *r, *q;
  if (cudaMalloc(&d, n * 8) || cudaMalloc(&r, n * 8) || cudaMalloc(&q, n * 8)) return 2;
  cudaMemcpy(d, h.data(), n * 8, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(n, d, r, q);
  std::vector<double> hr(n), hq(n);
  if (cudaMemcpy(hr.data(), r, n * 8, cudaMemcpyDeviceToHost) || cudaMemcpy(hq.data(), q, n * 8, cudaMemcpyDeviceToHost))
    return 3;
  long long most = 0, inside = 0, outside = 0;
  for (int i = 0; i < n; ++i) {
    long long a, b;
    std::memcpy(&a, &hr[i], 8);
    std::memcpy(&b, &hq[i], 8);
    if (h[i] > 1e-290 && h[i] < 1e290) {
      ++inside;
      most = std::max(most, std::llabs(a - b));
    } else if (a != b && !(std::isnan(hr[i]) && std::isnan(hq[i]))) {
      ++outside;
    }
  }
  std::printf("%d %lld %lld %lld\n", n, inside, most, outside);
  return 0;
}
"""


def test_reciprocal_is_within_one_unit_of_the_division(tmp_path):
    if not (os.path.exists(build.NVCC) or shutil.which(build.NVCC)):
        pytest.skip("no CUDA compiler here")
    src, exe = tmp_path / "r.cu", tmp_path / "r"
    src.write_text(PROGRAM)
    subprocess.run([build.NVCC, *build.ARCH, "-O3", "-std=c++17", "-I", build.CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    n, inside, most, outside = map(int, r.stdout.split())
    assert n > 1_000_000 and inside > 900_000
    assert most <= 1
    assert outside == 0
