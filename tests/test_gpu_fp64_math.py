"""The FP64 elementary functions of csrc/fp64_math.cuh against CUDA's own, over
the ranges that the walks use and at their edges: powers of two, arguments
around 1, the ends of the tables, zeros, subnormals, infinities and NaN.

The header states errors of at most 2 units in the last place (1.5 for exp);
CUDA's are at most 1 (2 for rsqrt), so the two differ by at most 4."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r'''
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "fp64_math.cuh"
using namespace dp;
__device__ double ulps(double a, double b) {  // |a - b| in units of b's last place
  if (isnan(a) && isnan(b)) return 0.0;
  if (a == b) return 0.0;
  if (!isfinite(a) || !isfinite(b)) return 1e30;
  const double u = nextafter(fabs(b), 1e308) - fabs(b);
  return fabs(a - b) / u;
}
__global__ void check(const double* x, int n, double* worst) {
  double w[8] = {0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double v = x[i];
    w[0] = fmax(w[0], ulps(f64::log(v), log(v)));
    const double e = fabs(v) < 1e3 ? v : 0.0;
    w[1] = fmax(w[1], ulps(f64::exp(e), exp(e)));
    w[1] = fmax(w[1], ulps(f64::exp(-e), exp(-e)));
    const double a = fabs(v);
    if (a > 1e-290 && a < 1e290) {
      w[2] = fmax(w[2], ulps(f64::rcp(v), 1.0 / v));
      w[3] = fmax(w[3], ulps(f64::rsqrt(a), rsqrt(a)));
      w[3] = fmax(w[3], ulps(f64::sqrt(a), sqrt(a)));
      const double p = f64::min_pos(a, 3.0), q = f64::max_pos(a, 3.0);
      if (p != fmin(a, 3.0) || q != fmax(a, 3.0) || f64::lt_pos(a, 3.0) != (a < 3.0)) w[6] = 1e30;
    }
    const double t = a <= 1.0 ? v : v - 2.0 * rint(0.5 * v);
    if (fabs(t) <= 1.0) {
      double s, c;
      f64::sincospi(t, &s, &c);  // absolute: units of 2^-53
      w[4] = fmax(w[4], fmax(fabs(s - sinpi(t)), fabs(c - cospi(t))) * 0x1p53);
    }
    const uint32_t k = uint32_t(i) * 2654435761u, l = k * 40503u + 17u;
    for (int h = 0; h < 32; h += 5)
      if (f64::uniform(k >> h, l) != u01(k >> h, l) || f64::uniform(0, l >> h) != u01(0, l >> h)) w[5] = 1e30;
    if (f64::from_int(int(k)) != double(int(k))) w[7] = 1e30;
  }
  for (int j = 0; j < 8; ++j)
    atomicMax(reinterpret_cast<unsigned long long*>(worst + j), (unsigned long long)__double_as_longlong(w[j]));
}
int main() {
  std::vector<double> x;
  for (double v : {0.0, -0.0, -1.0, 1.0, 5e-324, 1e-310, 2.2250738585072014e-308, 1.7e308, HUGE_VAL, -HUGE_VAL, HUGE_VAL - HUGE_VAL,
                   708.0, 709.9, -745.0, 0.75, 1.5, 2.0, 0.5})
    x.push_back(v);
  for (int j = 0; j < 512; ++j)  // the tables' edges and their neighbours
    for (double s : {1.0 + j / 512.0, (1.0 + j / 512.0) * 0.5, j / 64.0 - 4.0, j * 0.0027076061740622863})
      for (int d = -1; d <= 1; ++d) x.push_back(d < 0 ? nextafter(s, -1e9) : d ? nextafter(s, 1e9) : s);
  srand(1);
  for (int i = 0; i < 2000000; ++i) {
    const double u = (rand() + 0.5) / (RAND_MAX + 1.0), r = (rand() + 0.5) / (RAND_MAX + 1.0);
    x.push_back(i % 4 == 0 ? exp(-40.0 + 80.0 * u) : i % 4 == 1 ? 1.0 + (u - 0.5) * r * 0.1
                : i % 4 == 2 ? (u - 0.5) * 40.0 * r : u);
  }
  double *d, *w, h[8];
  cudaMalloc(&d, x.size() * 8);
  cudaMalloc(&w, 64);
  cudaMemset(w, 0, 64);
  cudaMemcpy(d, x.data(), x.size() * 8, cudaMemcpyHostToDevice);
  check<<<152, 128>>>(d, int(x.size()), w);
  if (cudaMemcpy(h, w, 64, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  for (int j = 0; j < 8; ++j) printf("%.3f ", h[j]);
  return 0;
}
'''


def test_against_cuda(tmp_path):
    import build
    src, exe = tmp_path / "check.cu", tmp_path / "check"
    src.write_text(SOURCE)
    subprocess.check_call([build.nvcc(), *build.ARCH, "-O2", "-std=c++17", "-I", build.SRC,
                           str(src), "-o", str(exe)])
    w = [float(v) for v in subprocess.check_output([str(exe)], timeout=120).split()]
    log, exp, rcp, root, trig, uniform, order, integer = w
    assert max(log, exp, rcp, root, trig) <= 4.0, w
    assert uniform == order == integer == 0.0, w
