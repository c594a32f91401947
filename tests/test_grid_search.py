"""The interval search of csrc/fp64_math.cuh, run on the host with the device's own
log: it ends, and with the right offset, at every node of a log-uniform energy grid
and up to two last places beside it, from every start near the node and from both ends.
The table's logs are the C library's and the lookups' are f64::log's, so the two differ
by a last place at some nodes; near 1 GeV, where the log is small against the grid's
spacing, that place is lost in the offset from the node below.

Offsets are (lx - x[i]) inv[i] with both factors rounded and the difference too: the
node is found to 3 halves of a last place of the larger of 1 and |log E| / width, in
widths (2 of them: the bound here)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "diffpumas.jl_gb300", "csrc")

SOURCE = r'''
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>
static inline long long __double_as_longlong(double x) { long long b; memcpy(&b, &x, 8); return b; }
static inline double __longlong_as_double(long long b) { double x; memcpy(&x, &b, 8); return x; }
static inline unsigned __float_as_uint(float x) { unsigned b; memcpy(&b, &x, 4); return b; }
static inline int __double2hiint(double x) { return int(__double_as_longlong(x) >> 32); }
static inline int __double2loint(double x) { return int(__double_as_longlong(x)); }
static inline double __hiloint2double(int h, int l) {
  return __longlong_as_double((long long)((unsigned long long)(unsigned)h << 32 | (unsigned)l));
}
static inline int __clzll(unsigned long long x) { return __builtin_clzll(x); }
#include "fp64_math.cuh"
using namespace dp;

int main() {
  long grids = 0, places = 0, split = 0, wrong = 0;
  const double lo[] = {1e-4, 3e-4, 1e-3, 2e-3, 1e-2, 0.05, 0.1, 0.5}, hi[] = {20.0, 1e2, 1e3, 1e4, 1e6, 1e8, 1e9, 1e10};
  for (double a : lo)
    for (double b : hi)
      for (int n : {2, 3, 5, 9, 17, 34, 64, 100, 146, 200, 201, 320, 641, 1601}) {
        ++grids;
        std::vector<double> E(n), x(n), inv(n, 0.0);
        for (int i = 0; i < n; ++i) x[i] = std::log(E[i] = a * std::pow(b / a, double(i) / double(n - 1)));
        for (int i = 0; i + 1 < n; ++i) inv[i] = 1.0 / (x[i + 1] - x[i]);
        for (int k = 0; k < n; ++k)
          for (int d = -2; d <= 2; ++d) {
            double e = E[k];
            for (int s = 0; s < std::abs(d); ++s) e = std::nextafter(e, d < 0 ? 0.0 : 1e300);
            if (!(e > E[0] && e < E[n - 1])) continue;  // the callers clamp
            const double lx = f64::log(e);
            if (d == 0 && lx != x[k]) ++split;
            for (int from : {k - 2, k - 1, k, k + 1, 0, n - 2}) {
              int i = from < 0 ? 0 : (from > n - 2 ? n - 2 : from);
              const double t = f64::grid_offset(x.data(), inv.data(), n, lx, i);
              ++places;
              const double tol = 2.0 * 2.3e-16 * std::fmax(1.0, std::fabs(lx) * inv[i]);
              const double off = double(((long double)lx - x[i]) / ((long double)x[i + 1] - x[i]));
              if (!(i >= 0 && i <= n - 2 && std::fabs(t - off) <= tol && t >= -tol && t <= 1.0 + tol)) ++wrong;
            }
          }
      }
  printf("%ld %ld %ld %ld\n", grids, places, split, wrong);
  return 0;
}
'''


def test_search_ends_at_every_node(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if cxx is None or not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("needs a host compiler and the CUDA headers")
    src, exe = tmp_path / "search.cpp", tmp_path / "search"
    src.write_text(SOURCE)
    subprocess.check_call([cxx, "-O1", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-I", include,
                           str(src), "-o", str(exe)])
    grids, places, split, wrong = map(int, subprocess.check_output([str(exe)], timeout=120).split())
    assert wrong == 0, (grids, places, wrong)
    assert split > 100, "the grids hold no node whose log the two sides round differently"


NAN_SOURCE = r'''
#include <cmath>
#include <cstdio>
#include <limits>
#include <vector>
#include "common.cuh"
int main() {
  int bad = 0;
  for (int n : {2, 3, 200}) {
    std::vector<double> x(n);
    for (int i = 0; i < n; ++i) x[i] = -7.0 + 0.1 * i;
    const double nan = std::numeric_limits<double>::quiet_NaN();
    for (double lx : {nan, -nan, -1e300, 1e300, -std::numeric_limits<double>::infinity(),
                      std::numeric_limits<double>::infinity()}) {
      volatile double v = lx;
      const int i = dp::uniform_interval(x.data(), n, v, x[0], 10.0);
      if (i < 0 || i > n - 2) ++bad;
    }
  }
  printf("%d\n", bad);
  return 0;
}
'''


def test_uniform_search_of_a_nan_stays_on_the_grid(tmp_path):
    """A double NaN converts to the lowest int (x86 and the device): the search of
    csrc/common.cuh read the grid from there on."""
    cxx = shutil.which("g++") or shutil.which("c++")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if cxx is None or not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("needs a host compiler and the CUDA headers")
    src, exe = tmp_path / "nan.cpp", tmp_path / "nan"
    src.write_text(NAN_SOURCE)
    subprocess.check_call([cxx, "-O1", "-std=c++17", "-I", CSRC, "-I", include, str(src), "-o", str(exe)])
    assert int(subprocess.check_output([str(exe)], timeout=60)) == 0
