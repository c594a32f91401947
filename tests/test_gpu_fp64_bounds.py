"""Error bounds of csrc/fp64_math.cuh against the host's extended precision (long double),
and its exact operations bit for bit.

The bounds, in units of the result's last place, from the roundings of each form:
 log    2     constant of log 2, table value, their sum and the result, half a unit each
              where the sum cancels most (x just below 3/4)
 exp    1.25  table value and result; the polynomial's term is below 2^-8 of the result
 rcp    0.75  the result; the residual is formed exactly and its cube is below 2^-60
 rsqrt  1.25  the residual (one rounding, halved) and the result
 div    1.75  rcp's error, doubled at most by the quotient's binade, and the result
 sqrt   2.125 rsqrt's 1.5 2^-53 in all and the result
 1/(beta gamma) 2.25: rsqrt's, and half of the roundings of x + 2 and x (x + 2); its
              derivative 12: three times the value's 2.5 2^-53, and four roundings"""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r'''
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "fp64_math.cuh"
using namespace dp;
typedef long double LD;
enum { LOG, EXP, RCP, RSQRT, SQRT, DIV, IBG, DIBG, NF };
__global__ void eval(const double* x, const double* b, int n, double* o) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double v = x[i];
    double d;
    o[LOG * n + i] = f64::log(v);
    o[EXP * n + i] = f64::exp(log(v) * 17.0);
    o[RCP * n + i] = f64::rcp(v);
    o[RSQRT * n + i] = f64::rsqrt(v);
    o[SQRT * n + i] = f64::sqrt(v);
    o[DIV * n + i] = f64::div(v, b[i]);
    o[IBG * n + i] = f64::inv_beta_gamma(v, &d);
    o[DIBG * n + i] = d;
  }
}
__global__ void args(const double* x, int n, double* e) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) e[i] = log(x[i]) * 17.0;
}
__global__ void exact(const double* x, const double* b, const float* f, int n, double* q, double* w) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    q[i] = f64::div_rn(x[i], b[i], __drcp_rn(b[i]));
    w[i] = f64::widen(f[i]);
  }
}
static double ulps(double a, LD t) {
  const double r = double(t);
  return std::isfinite(a) ? double(fabsl(LD(a) - t) / LD(nextafter(fabs(r), HUGE_VAL) - fabs(r))) : 1e30;
}
template <class T> static T* up(const std::vector<T>& v) {
  T* d;
  cudaMalloc(&d, v.size() * sizeof(T));
  cudaMemcpy(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
  return d;
}
int main() {
  std::vector<double> x, b;
  srand(3);
  auto u = [] { return (rand() + 0.5) / (RAND_MAX + 1.0); };
  for (int i = 0; i < 200000; ++i) {
    x.push_back(i % 3 == 0 ? exp(40.0 * (u() - 0.5)) : i % 3 == 1 ? 0.3 + 2.0 * u() : 1.0 + (u() - 0.5) * 0.01);
    b.push_back((i & 1 ? -1.0 : 1.0) * exp(40.0 * (u() - 0.5)));
  }
  const int n = int(x.size());
  std::vector<float> f;
  for (uint32_t k = 0; k < uint32_t(n); ++k) {  // all exponents, both signs, the classes among them
    const uint32_t bits = k < 1024 ? (k % 512) << 23 | (k < 512 ? 0u : 0x2345u) : k * 2654435761u;
    float v;
    memcpy(&v, &bits, 4);
    f.push_back(v);
  }
  double *dx = up(x), *db = up(b), *o = up(std::vector<double>(size_t(NF) * n)), *e = up(x), *q = up(x), *w = up(x);
  float* df = up(f);
  eval<<<152, 128>>>(dx, db, n, o);
  args<<<152, 128>>>(dx, n, e);
  exact<<<152, 128>>>(dx, db, df, n, q, w);
  std::vector<double> r(size_t(NF) * n), he(n), hq(n), hw(n);
  if (cudaMemcpy(r.data(), o, r.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  cudaMemcpy(he.data(), e, 8 * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(hq.data(), q, 8 * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(hw.data(), w, 8 * n, cudaMemcpyDeviceToHost);
  double m[NF] = {0}, wrong = 0;
  for (int i = 0; i < n; ++i) {
    const LD v = x[i], g = sqrtl(v * (v + 2));
    const LD t[NF] = {logl(v), expl(LD(he[i])), 1 / v, 1 / sqrtl(v), sqrtl(v), v / LD(b[i]), 1 / g, -(v + 1) / (g * g * g)};
    for (int k = 0; k < NF; ++k) m[k] = fmax(m[k], ulps(r[size_t(k) * n + i], t[k]));
    const double ww = double(f[i]), qq = x[i] / b[i];
    if (memcmp(&hq[i], &qq, 8)) ++wrong;
    if (std::isnan(ww) ? !std::isnan(hw[i]) : memcmp(&hw[i], &ww, 8) != 0) ++wrong;
  }
  for (double v : m) printf("%.4f ", v);
  // outside of the quick form: the clamp of beta, negative energies, squares that overflow
  std::vector<double> y = {0.0, 1e-300, 9.9e-13, 1e-12, 1.1e-12, -1e-13, -0.5, -1.5, -3.0, -1e200, 9.9e99, 1.1e100, 1e160, 1e300, HUGE_VAL, -HUGE_VAL};
  const int k = int(y.size());
  double *dy = up(y), *o2 = up(std::vector<double>(size_t(NF) * k));
  eval<<<1, 32>>>(dy, dy, k, o2);
  std::vector<double> s(size_t(NF) * k);
  cudaMemcpy(s.data(), o2, s.size() * 8, cudaMemcpyDeviceToHost);
  double far = 0;
  for (int i = 0; i < k; ++i) {  // the reference's operations
    const double g = 1.0 + y[i], b2 = 1.0 - 1.0 / (g * g), t = 1.0 / (sqrt(b2 > 1e-12 ? b2 : 1e-12) * g), a = s[IBG * k + i];
    // below 1e-11 the quick form keeps the digits that 1 - 1/g^2 loses
    far = fmax(far, t == a ? 0.0 : fabs(a - t) / fabs(t) / (fabs(y[i]) < 1e-11 && y[i] >= 1e-12 ? 1e12 : 1.0));
    if (!std::isfinite(s[DIBG * k + i])) far = 1e30;
  }
  printf("%g %g\n", far, wrong);
  return 0;
}
'''


def test_bounds(tmp_path):
    import build
    src, exe = tmp_path / "bounds.cu", tmp_path / "bounds"
    src.write_text(SOURCE)
    subprocess.check_call([build.nvcc(), *build.ARCH, "-O2", "-std=c++17", "-I", build.SRC, str(src), "-o", str(exe)])
    v = [float(x) for x in subprocess.check_output([str(exe)], timeout=120).split()]
    names = ("log", "exp", "rcp", "rsqrt", "sqrt", "div", "inv_beta_gamma", "its derivative")
    bounds = (2.0, 1.25, 0.75, 1.25, 2.125, 1.75, 2.25, 12.0)
    print(dict(zip(names, v)))
    assert all(x <= y for x, y in zip(v, bounds)), dict(zip(names, v))
    assert v[8] <= 1e-14 and v[9] == 0.0, v
