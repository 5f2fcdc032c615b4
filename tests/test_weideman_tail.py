"""The single-precision terms of w_weideman_fast (faddeeva.cuh) on the CPU: what
they move w by, apart from every other rounding of the series.  The remaining
recurrence runs in 80 bits from the single-precision terms and from the exact
ones.  Bound: 2^-58 of |w|; in quadrature with the double-precision form's
smallest rms error, 1.3e-16, that is 0.04 %."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cetasim_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <random>
#include "faddeeva_table.cpp"
using namespace cg;
int main() {
  weideman_table_init(&h_weideman);
  const WeidemanTable& T = h_weideman;
  constexpr int N = kWeidemanN, K = kWeidemanTail;
  std::mt19937_64 g(3);
  std::uniform_real_distribution<double> u(0, 1);
  long double worst = 0;
  for (int i = 0; i < 400000; ++i) {
    // |z| < 30, every other point near the real axis
    const double m = 30 * std::pow(u(g), 1.5), t = 1.5707963267948966 * u(g);
    const double x = i & 1 ? m : m * std::cos(t), y = i & 1 ? std::pow(10, -8 + 8 * t / 1.5708) : m * std::sin(t);
    if (x * x + y * y >= 900) continue;
    cplx rden;
    const cplx Z = weideman_map(x, y, T.L, &rden);
    const double r = 2 * Z.re, s = std::fma(Z.re, Z.re, Z.im * Z.im);
    const float rf = (float)r, sf = (float)s;
    float f2 = T.t[0], f1 = std::fmaf(rf, f2, T.t[1]);
    long double e2 = T.a[0], e1 = r * e2 + T.a[1];
    for (int n = 2; n < K; ++n) {
      const float f = std::fmaf(rf, f1, std::fmaf(-sf, f2, T.t[n]));
      const long double e = r * e1 - s * e2 + T.a[n];
      f2 = f1; f1 = f; e2 = e1; e1 = e;
    }
    long double b1 = e1 - f1, b2 = e2 - f2;  // the recurrence is linear
    for (int n = K; n < N - 1; ++n) {
      const long double b = r * b1 - s * b2;
      b2 = b1; b1 = b;
    }
    const long double p = hypotl(b1 * Z.re - s * b2, b1 * Z.im);
    const cplx w = w_weideman(x, y);
    worst = fmaxl(worst, 2 * p * ((long double)rden.re * rden.re + (long double)rden.im * rden.im) /
                             hypotl(w.re, w.im));
  }
  std::printf("%.6Le\n", worst);
}
"""


def test_single_precision_terms_are_below_rounding(tmp_path):
    src, exe = tmp_path / "tail.cpp", tmp_path / "tail"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-march=native", "-std=c++17", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    worst = float(subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout)
    assert 0 < worst <= 2.0 ** -58
