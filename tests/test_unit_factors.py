"""Unit factors in FP32 (csrc/ms_unit.h): the pair chosen for an angle, and
what choosing it costs.

Every twiddle and propagator factor of a set-up goes through this function (a
few thousand to some ten thousand a grid), so it must not take more than a few
library calls.  The limit is relative to this host's own atan2: an exhaustive
choice by inverse functions takes nine of them and as many remainders."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include <chrono>
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include "ms_unit.h"
template <class F> double ns(F f) {
  double best = 1e30;
  for (int rep = 0; rep < 5; ++rep) {
    auto t0 = std::chrono::steady_clock::now();
    for (int i = 0; i < 200000; ++i) f(std::cos(i * 3e-5), std::sin(i * 3e-5));
    best = std::fmin(best, std::chrono::duration<double, std::nano>(std::chrono::steady_clock::now() - t0).count() / 200000);
  }
  return best;
}
int main() {
  volatile float sink = 0;
  double modulus = 0, angle = 0;
  for (int n : {7, 12, 64, 343, 600, 1024, 4096})
    for (int m = 0; m < n; ++m) {
      const double a = 6.283185307179586 * m / n;
      float x, y;
      ms::unit_fp32(std::cos(a), std::sin(a), &x, &y);
      modulus = std::fmax(modulus, std::fabs((double)x * x + (double)y * y - 1));
      angle = std::fmax(angle, std::fabs(std::remainder(std::atan2((double)y, (double)x) - a, 6.283185307179586)));
    }
  const double t = ns([&](double c, double s) { float x, y; ms::unit_fp32(c, s, &x, &y); sink = sink + x + y; });
  const double u = ns([&](double c, double s) { sink = sink + (float)std::atan2(s, c); });
  const double v = ns([&](double c, double s) { sink = sink + (float)(s + c); });
  std::printf("%g %g %g %g %g\n", modulus, angle, t, u, v);
}
"""


def test_unit_factors(tmp_path):
    src, exe = tmp_path / "unit.cpp", tmp_path / "unit"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I" + os.path.join(ROOT, "cudamultislice_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True, timeout=120).stdout
    modulus, angle, t, t_atan2, t_loop = map(float, out.split())
    # no worse than the rounded pair (half an ulp of 2^-24 each, times cos + sin,
    # twice for the square) weighed with its angle; one ulp and a half each
    assert modulus < 2.0 ** -23 and angle < 1.5 * 2.0 ** -23, out
    assert t - t_loop < 6 * (t_atan2 - t_loop), out
