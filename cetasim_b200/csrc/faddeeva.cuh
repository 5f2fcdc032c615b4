// FP64 Faddeeva function w(z) = exp(-z^2) erfc(-i z) for the sm_100a kernels.
//
// Replaces the vendored Faddeeva::w that the reference calls inside
// Bunch::BassettiErskine1 (Bunch.cpp:147, Bunch.cpp:150).  The algorithm here
// is this project's own, built from published methods:
//
//   * Weideman's rational series (J.A.C. Weideman, "Computation of the complex
//     error function", SIAM J. Numer. Anal. 31 (1994) 1497-1518) with N = 40
//     terms for |z| < 8: one complex Horner chain, no branches.  The 40
//     coefficients are computed at library load by a long-double DFT of
//     exp(-t^2)(L^2 + t^2), t = L tan(theta/2), exactly as the paper defines
//     them, and live in __constant__ memory.
//   * The Laplace continued fraction (Gauss-Hermite J-fraction) for |z| >= 8,
//     with a depth chosen per |z| band (8 terms for |z| >= 12, 12 terms below);
//     near the real axis the exponentially small Stokes term exp(-z^2), which
//     no finite depth of the fraction carries, is added back.
//
// Two entry points:
//   w_quadrant1(x, y)  x, y >= 0 -- the field-kick path.  Region switching is
//                      warp-uniform in practice (see be_field.cuh): a warp
//                      takes the Weideman branch unless all its lanes are far.
//   w_general(x, y)    any z, including the lower half plane (reflection
//                      w(z) = 2 exp(-z^2) - w(-z)), infinities and NaN, with
//                      per-component accuracy near both axes.  Used for the
//                      known-answer test and for callers that need a general
//                      w(z).
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define CG_HD __host__ __device__ __forceinline__
#else
#define CG_HD inline
#endif

namespace cg {

constexpr int kWeidemanN = 40;
// The coefficients of Z^28 .. Z^39 are below 2e-11 of the leading one, so
// single precision in their part of the series moves w by at most 1.4e-18 |w| =
// 2^-59 |w| for |z| < 30 (14 terms: 1.4e-17): w_weideman_fast sums them in the
// FP32 pipe.  Against binary128 the rms errors are those of the all-FP64 series
// to 0.1 % in fourteen ranges of z (4.0e-16 of |w| for |z| < 1, 1.3e-16 for
// 8 < |z| < 30, 2.4e-16 for 5 < x < 8 near the real axis, where 14 terms left
// 0.7 % more in places).
constexpr int kWeidemanTail = 12;

struct alignas(128) WeidemanTable {  // whole lines of the constant cache
  double a[kWeidemanN];  // highest power first (Horner order)
  double L;
  float t[kWeidemanTail];  // the first of a in single precision
};

#ifdef __CUDACC__
// One copy per translation unit (the library is built without relocatable
// device code); upload_weideman_table() fills the copy of kernels.cu, which
// holds every kernel that evaluates w(z).
static __constant__ WeidemanTable c_weideman;
#endif
extern WeidemanTable h_weideman;  // host copy (filled by weideman_table_init)

// Computes the Weideman coefficients (host, once).
void weideman_table_init(WeidemanTable* t);

CG_HD const WeidemanTable& weideman_table() {
#if defined(__CUDA_ARCH__)
  return c_weideman;
#else
  return h_weideman;
#endif
}

constexpr double kInvSqrtPi = 0.56418958354775628695;  // 1/sqrt(pi)
constexpr double kTwoInvSqrtPi = 1.1283791670955125739;  // 2/sqrt(pi)

struct cplx {
  double re, im;
};

CG_HD cplx cmul(cplx a, cplx b) {
  return {fma(a.re, b.re, -a.im * b.im), fma(a.re, b.im, a.im * b.re)};
}

// a / b with the scaling of Smith's algorithm (no overflow for large |b|).
CG_HD cplx cdiv(cplx a, cplx b) {
  if (fabs(b.re) >= fabs(b.im)) {
    double r = b.im / b.re, d = 1.0 / fma(b.im, r, b.re);
    return {fma(a.im, r, a.re) * d, fma(-a.re, r, a.im) * d};
  } else {
    double r = b.re / b.im, d = 1.0 / fma(b.re, r, b.im);
    return {fma(a.re, r, a.im) * d, fma(a.im, r, -a.re) * d};
  }
}

// Weideman rational series, valid for Im z >= 0.
CG_HD cplx w_weideman(double x, double y) {
  const WeidemanTable& T = weideman_table();
  const double L = T.L;
  // iz = -y + i x;  den = L - iz = (L + y) - i x;  num = L + iz = (L - y) + i x
  cplx den = {L + y, -x};
  cplx num = {L - y, x};
  // Z = num / den.  |den| >= L > 0 in the upper half plane.
  double inv = 1.0 / fma(den.re, den.re, den.im * den.im);
  cplx Z = {fma(num.re, den.re, num.im * den.im) * inv,
            fma(num.im, den.re, -num.re * den.im) * inv};
  cplx p = {T.a[0], 0.0};
#pragma unroll
  for (int n = 1; n < kWeidemanN; ++n) {
    cplx q = cmul(p, Z);
    p = {q.re + T.a[n], q.im};
  }
  // 1/den = conj(den) * inv
  cplx rden = {den.re * inv, -den.im * inv};
  cplx rden2 = cmul(rden, rden);
  cplx t = cmul(p, rden2);
  return {fma(2.0, t.re, kInvSqrtPi * rden.re), fma(2.0, t.im, kInvSqrtPi * rden.im)};
}

CG_HD cplx cmuladd(cplx a, cplx b, cplx z) {  // a + b z
  return {fma(b.re, z.re, fma(-b.im, z.im, a.re)), fma(b.re, z.im, fma(b.im, z.re, a.im))};
}

// Laplace continued fraction of fixed depth, Im z >= 0, |z| large.
template <int DEPTH>
CG_HD cplx w_cfrac(double x, double y) {
  cplx t = {x, y};
#pragma unroll
  for (int k = DEPTH; k >= 1; --k) {
    cplx q = cdiv({0.5 * k, 0.0}, t);
    t = {x - q.re, y - q.im};
  }
  cplx r = cdiv({0.0, kInvSqrtPi}, t);
  return r;
}

// exp(-z^2) for z = x + i y, returning 0 when the modulus underflows (so that
// an overflowing phase 2xy never turns 0 into NaN).
CG_HD cplx cexp_mz2(double x, double y) {
  double re = (y - x) * (y + x);  // Re(-z^2) = y^2 - x^2
  if (re < -745.2) return {0.0, 0.0};
  double m = exp(re);
  double s, c;
  sincos(-2.0 * x * y, &s, &c);
  return {m * c, m * s};
}

// exp(-q) for q >= 0 without a branch, so that a caller's other arithmetic is
// scheduled beside it (the library exp branches on its argument's range):
// argument reduction q = -(n ln 2 + f) with ln 2 in two parts (W. J. Cody and
// W. Waite, Software Manual for the Elementary Functions, 1980), |f| <= ln 2 /
// 2, and the Taylor series of e^f to f^13 (remainder 5e-18).  Beyond q = 708
// (and for a NaN) the value at 708, 3e-308, in place of the subnormal range.
CG_HD double exp_neg(double q) {
  q = fmin(q, 708.0);
  const double magic = 6755399441055744.0;  // 1.5 2^52: the sum's low word is the integer
  const double t = fma(q, -1.4426950408889634074, magic);
  const double n = t - magic;
  double f = fma(n, -0.69314718036912381649, -q);   // ln 2, upper 32 bits
  f = fma(n, -1.9082149292705877e-10, f);           // ln 2 - the upper part
  double p = 1.0 / 6227020800.0;
  p = fma(p, f, 1.0 / 479001600.0);
  p = fma(p, f, 1.0 / 39916800.0);
  p = fma(p, f, 1.0 / 3628800.0);
  p = fma(p, f, 1.0 / 362880.0);
  p = fma(p, f, 1.0 / 40320.0);
  p = fma(p, f, 1.0 / 5040.0);
  p = fma(p, f, 1.0 / 720.0);
  p = fma(p, f, 1.0 / 120.0);
  p = fma(p, f, 1.0 / 24.0);
  p = fma(p, f, 1.0 / 6.0);
  p = fma(p, f, 0.5);
  p = fma(p, f, 1.0);
  p = fma(p, f, 1.0);
#if defined(__CUDA_ARCH__)
  return __hiloint2double(__double2hiint(p) + (__double2loint(t) << 20), __double2loint(p));
#else
  return ldexp(p, (int)n);
#endif
}

// First-quadrant kernel path (x >= 0, y >= 0): ~1e-15 relative to |w|.
CG_HD cplx w_quadrant1(double x, double y) {
  double r2 = fma(x, x, y * y);
  if (r2 < 64.0) return w_weideman(x, y);
  cplx w = (r2 < 144.0) ? w_cfrac<12>(x, y) : w_cfrac<8>(x, y);
  if (y < 1.0) {  // Stokes term near the real axis (negligible elsewhere)
    cplx e = cexp_mz2(x, y);
    w.re += e.re;
    w.im += e.im;
  }
  return w;
}

// 1/d for 1e-300 < d < 1e300 (on the host, whose seed is single precision, 1e-30
// to 3e38) by Newton-Raphson refinement of an approximate
// seed (two steps, r <- r + r (1 - d r): 2^-20 -> 2^-40 -> rounding level,
// within about an ulp of the correctly rounded quotient).  The seed is the
// double-precision reciprocal approximation: 18 cycles, against 60 for a
// conversion to float, a reciprocal there and the conversion back.
CG_HD double recip_newton(double d) {
#if defined(__CUDA_ARCH__)
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
#else
  double r = (double)(1.0f / (float)d);
#endif
  double e = fma(-d, r, 1.0);
  r = fma(r, e, r);
  e = fma(-d, r, 1.0);
  return fma(r, e, r);
}

// w(z) from the series p and rden = 1/(L - iz).
CG_HD cplx weideman_from_sum(cplx p, cplx rden) {
  cplx rden2 = cmul(rden, rden);
  cplx t = cmul(p, rden2);
  return {fma(2.0, t.re, kInvSqrtPi * rden.re), fma(2.0, t.im, kInvSqrtPi * rden.im)};
}

// The map z -> Z = (L + iz)/(L - iz) of Weideman's series and rden = 1/(L - iz).
CG_HD cplx weideman_map(double x, double y, double L, cplx* rden) {
  const cplx den = {L + y, -x};
  const cplx num = {L - y, x};
  const double inv = recip_newton(fma(den.re, den.re, den.im * den.im));
  *rden = {den.re * inv, -den.im * inv};
  return {fma(num.re, den.re, num.im * den.im) * inv, fma(num.im, den.re, -num.re * den.im) * inv};
}

// Weideman's series at NW points with Knuth's evaluation of a polynomial with
// real coefficients at a complex point (The Art of Computer Programming,
// vol. 2, 4.6.4): with r = 2 Re Z and s = |Z|^2, the remainder of p modulo
// Z^2 - r Z + s (which vanishes at Z) follows from the real recurrence
// b_k = c_k + r b_{k+1} - s b_{k+2}, and p(Z) = b_1 Z + c_0 - s b_2: two FMAs
// per term instead of the four FP64 instructions of a complex Horner step.
// A rounding of b_k acts on p as the same change of c_k times Z^k, and
// |b_k| stays below 1e-10 down to k = 28, so the first kWeidemanTail steps run
// in single precision and 24 of the 76 FP64 operations per point go to the FP32
// pipe, which the kick leaves idle.  The NW recurrences run side by side: each
// is one FMA latency per term.  For |z| < 30 in the first quadrant within 2e-15
// of w relative to |w| (the form the throughput kernels use).
template <int NW>
CG_HD void w_weideman_fast(const double (&x)[NW], const double (&y)[NW], cplx (&w)[NW]) {
  const WeidemanTable& T = weideman_table();
  cplx Z[NW], rden[NW];
  double r[NW], s[NW], b1[NW], b2[NW];
  float rf[NW], sf[NW], f1[NW], f2[NW];
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    Z[i] = weideman_map(x[i], y[i], T.L, &rden[i]);
    r[i] = 2.0 * Z[i].re;
    s[i] = fma(Z[i].re, Z[i].re, Z[i].im * Z[i].im);
    rf[i] = (float)r[i];
    sf[i] = (float)s[i];
    // c_m = a[N - 1 - m]: b_{N-1} = a[0], b_{N-2} = a[1] + r b_{N-1}
    f2[i] = T.t[0];
    f1[i] = fmaf(rf[i], f2[i], T.t[1]);
  }
#pragma unroll
  for (int n = 2; n < kWeidemanTail; ++n)
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      const float b = fmaf(rf[i], f1[i], fmaf(-sf[i], f2[i], T.t[n]));
      f2[i] = f1[i];
      f1[i] = b;
    }
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    b1[i] = (double)f1[i];
    b2[i] = (double)f2[i];
  }
#pragma unroll
  for (int n = kWeidemanTail; n < kWeidemanN - 1; ++n)  // b_k, k = N - 1 - n, down to b_1
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      const double b = fma(r[i], b1[i], fma(-s[i], b2[i], T.a[n]));
      b2[i] = b1[i];
      b1[i] = b;
    }
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    const cplx p = {fma(b1[i], Z[i].re, fma(-s[i], b2[i], T.a[kWeidemanN - 1])), b1[i] * Z[i].im};
    w[i] = weideman_from_sum(p, rden[i]);
  }
}

// The kick kernels' first-quadrant path for the two w(z) of a point:
// Weideman's expansion up to |z| = 30, where it stays within 3e-14 of w
// relative to |w| (the real-axis region included), the continued fraction
// beyond.  Beam particles and ions sit within a few tens of sigma of the
// other beam, so every lane of a warp takes the same branch and the two w(z)
// of a kick run side by side.
CG_HD void w_quadrant1_wide2(const double (&x)[2], const double (&y)[2], cplx (&w)[2]) {
  if (fmax(fma(x[0], x[0], y[0] * y[0]), fma(x[1], x[1], y[1] * y[1])) < 900.0) {
    w_weideman_fast<2>(x, y, w);
  } else {
    for (int i = 0; i < 2; ++i) {
      const double xi[1] = {x[i]}, yi[1] = {y[i]};
      cplx wi[1];
      if (fma(x[i], x[i], y[i] * y[i]) < 900.0) {
        w_weideman_fast<1>(xi, yi, wi);
        w[i] = wi[0];
      } else {
        w[i] = w_cfrac<8>(x[i], y[i]);
      }
    }
  }
}

// scale * w(z) for 0 <= |z| < 30 in the first quadrant with a short dependent
// chain, for the ion walk, where each step waits for the one before it: the
// powers of Z by their remainder modulo 4 as four recurrences in Z^4 side by
// side (9 steps instead of 39; two at a time would leave the FP64 pipe idle
// half of the steps' latency, more would only add operations), and everything
// that multiplies the series (2 scale / (L - iz)^2) prepared while it is
// summed.  A step of the walk around it takes 600 cycles of one warp per
// sub-partition, 900 with the plain recurrence, 670 in Estrin's form.
CG_HD cplx weideman_scaled(double x, double y, double scale) {
  const WeidemanTable& T = weideman_table();
  constexpr int N = kWeidemanN;
  static_assert(N % 4 == 0, "four equal parts");
  cplx rden;
  const cplx Z = weideman_map(x, y, T.L, &rden);
  const cplx Z2 = cmul(Z, Z);
  const cplx v = cmul(Z2, Z2);
  const double r = 2.0 * v.re, s = fma(v.re, v.re, v.im * v.im);
  // c_m = a[N - 1 - m]; part k holds c_k, c_{k+4}, ...
  double b1[4], b2[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    b2[k] = T.a[3 - k];
    b1[k] = fma(r, b2[k], T.a[7 - k]);
  }
#pragma unroll
  for (int n = 2; n < N / 4 - 1; ++n)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double b = fma(r, b1[k], fma(-s, b2[k], T.a[4 * n + 3 - k]));
      b2[k] = b1[k];
      b1[k] = b;
    }
  cplx P[4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    P[k] = {fma(b1[k], v.re, fma(-s, b2[k], T.a[N - 1 - k])), b1[k] * v.im};
  const cplx p = cmuladd(cmuladd(P[0], P[1], Z), cmuladd(P[2], P[3], Z), Z2);
  const cplx rden2 = cmul(rden, rden);
  const double s2 = 2.0 * scale, s1 = kInvSqrtPi * scale;
  const cplx R = {rden2.re * s2, rden2.im * s2}, C = {rden.re * s1, rden.im * s1};
  return {fma(p.re, R.re, fma(-p.im, R.im, C.re)), fma(p.re, R.im, fma(p.im, R.re, C.im))};
}

// Near-real-axis strip (0 <= y < 0.5): shifted trapezoidal rule for
// (i/pi) Int exp(-t^2)/(z - t) dt plus the residue of the pole at t = z
// (Chiarella & Reichel 1968; Matta & Reichel 1971).  Every term of the real
// part is non-negative, so Re w keeps full relative accuracy even where it is
// exponentially smaller than Im w.
CG_HD cplx w_axis_strip(double x, double y) {
  const double h = 0.45;
  const double d = x - 0.5 * h;  // Re z sits midway between two nodes
  const double tmax = 6.2;       // exp(-6.2^2) = 2e-17
  int n0 = (int)floor((-tmax - d) / h);
  int n1 = (int)ceil((tmax - d) / h);
  double sre = 0.0, sim = 0.0;
  for (int n = n0; n <= n1; ++n) {
    double t = fma((double)n, h, d);
    double g = exp(-t * t);
    double u = x - t;
    double den = fma(u, u, y * y);
    // g / (z - t) = g (u - i y) / den ; times i h/pi -> (h/pi) g (y + i u)/den
    double f = g / den;
    sre = fma(f, y, sre);
    sim = fma(f, u, sim);
  }
  const double hpi = h * 0.31830988618379067154;  // h/pi
  cplx w = {hpi * sre, hpi * sim};
  // residue term 2 exp(-z^2) / (1 - exp(-2 pi i (z - d)/h)),
  // (z - d)/h = 1/2 + i y/h  =>  exp(-2 pi i (z-d)/h) = -exp(2 pi y/h)
  cplx e = cexp_mz2(x, y);
  double den = 1.0 + exp(6.283185307179586477 * y / h);
  w.re += 2.0 * e.re / den;
  w.im += 2.0 * e.im / den;
  return w;
}

// Upper half plane, x >= 0 (after the reflection x -> -x).
CG_HD cplx w_upper_right(double x, double y) {
  if (isinf(x) || isinf(y)) return {0.0, 0.0};
  if (x == 0.0 && y == 0.0) return {1.0, 0.0};
  double r2 = fma(x, x, y * y);
  if (!(r2 < 64.0)) {
    if (r2 > 1e24 || isinf(r2)) {
      // w ~ i/(sqrt(pi) z) (relative error 1/(2|z|^2) < 1e-24)
      cplx w = cdiv({0.0, kInvSqrtPi}, {x, y});
      if (y < 1.0) {
        cplx e = cexp_mz2(x, y);
        w.re += e.re;
        w.im += e.im;
      }
      return w;
    }
    return w_quadrant1(x, y);
  }
  if (x < 0.05) {
    // Taylor series in x about z0 = iy.  w(z0) = erfcx(y) is real, and the
    // derivatives follow w' = -2 z w + 2i/sqrt(pi), w^(n+1) = -2 z w^(n) -
    // 2n w^(n-1); at z0 = iy even derivatives are real and odd ones purely
    // imaginary, so Re w sums the even terms and Im w the odd ones, each
    // with full relative accuracy (Im w -> 0 linearly in x).
    double ex = w_weideman(0.0, y).re;
    double dm1 = ex;                              // w(z0)       (real)
    double d = kTwoInvSqrtPi - 2.0 * y * ex;      // w'(z0) / i  (real coefficient)
    double re = ex, im = x * d;
    double xn = x, fact = 1.0;
    // d_n stored as a real coefficient c_n with w^(n) = i^(n mod 2) c_n, so the
    // recurrence in real arithmetic reads c_{n+1} = s_n 2 y c_n - 2 n c_{n-1}
    // with s_n = +1 for n odd, -1 for n even.
#pragma unroll 1
    for (int n = 1; n < 18; ++n) {
      double s = (n & 1) ? 2.0 * y : -2.0 * y;
      double dn1 = s * d - 2.0 * n * dm1;
      dm1 = d;
      d = dn1;
      xn *= x;
      fact *= (double)(n + 1);
      double term = d * xn / fact;
      if ((n + 1) & 1) im += term; else re += term;
    }
    return {re, im};
  }
  if (y < 0.5 && x > 2.5) return w_axis_strip(x, y);
  return w_weideman(x, y);
}

// General w(z) for any complex z (NaN in -> NaN out).
CG_HD cplx w_general(double x, double y) {
  // NaN in gives NaN out, except that w(iy) stays real for x = 0
  if (isnan(x) || isnan(y)) return {NAN, x == 0.0 ? 0.0 : NAN};
  if (y >= 0.0) {
    if (x >= 0.0) return w_upper_right(x, y);
    cplx w = w_upper_right(-x, y);  // w(-conj z) = conj w(z)
    return {w.re, -w.im};
  }
  // lower half plane: w(z) = 2 exp(-z^2) - w(-z), -z in the upper half plane
  double mx = -x, my = -y;
  cplx wm;
  if (mx >= 0.0) {
    wm = w_upper_right(mx, my);
  } else {
    cplx t = w_upper_right(-mx, my);
    wm = {t.re, -t.im};
  }
  if (isinf(x) || isinf(y)) {
    if (isinf(y) && x == 0.0) return {INFINITY, 0.0};
    return {NAN, NAN};
  }
  double re = (y - x) * (y + x);  // Re(-z^2)
  if (re < -745.2) return {-wm.re, -wm.im};
  if (re > 709.7) {
    double s, c;
    sincos(-2.0 * x * y, &s, &c);
    return {c == 0.0 ? 0.0 : copysign(INFINITY, c), s == 0.0 ? 0.0 : copysign(INFINITY, s)};
  }
  cplx e = cexp_mz2(x, y);
  return {2.0 * e.re - wm.re, 2.0 * e.im - wm.im};
}

}  // namespace cg
