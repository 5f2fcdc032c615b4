// Normal draws and the RF phase on the device, written without branches so
// that the three pairs of a particle interleave.  One translation unit
// (kernels.cu) includes this header: its constants live in that unit's
// constant bank, where an FP64 instruction reads them as an operand.
#pragma once
#include "track_math.cuh"

namespace cg {

// whole lines of the constant cache (8 bytes off one, the turn's tail takes 506 us
// for 1.74e7 particles instead of 488)
struct alignas(128) NormalConst {
  double atanh_c[7];  // (atanh(s) / s - 1) / s^2 in s^2 <= 0.0295
  double sin_c[6];    // (sin(y) / y - 1) / y^2 in y^2, |y| <= pi / 4
  double cos_c[6];    // (cos(y) - 1 + y^2 / 2) / y^4 in y^2
  double ln2_hi, ln2_lo;  // -2 ln 2, the first with 32 bits: exact times an exponent
  double pio2_hi, pio2_lo;  // pi / 2, the first with 33 bits
};
// Chebyshev interpolation of the three functions in 60 digits, errors 5e-18,
// 1.3e-17 and 5e-19 relative to the function.
static __constant__ NormalConst c_norm = {
    {0.07309671726756307, 0.07665743617932867, 0.09091448091741543, 0.11111105518908294,
     0.14285714313285103, 0.19999999999949095, 0.3333333333333335},
    {1.5918115263265974e-10, -2.505113165023518e-08, 2.7557316101617874e-06,
     -0.00019841269836756774, 0.008333333333330948, -0.16666666666666666},
    {-1.1382623647474603e-11, 2.087614614655861e-09, -2.7557317271145144e-07,
     2.480158729876456e-05, -0.0013888888888887398, 0.041666666666666664},
    -0x1.62e42fee00000p+0, -0x1.a39ef35793c76p-32, 0x1.921fb54400000p+0, 0x1.0b4611a626331p-34};

template <int N>
__device__ __forceinline__ double norm_poly(const double (&a)[N], double x) {
  double p = a[0];
#pragma unroll
  for (int k = 1; k < N; ++k) p = fma(p, x, a[k]);
  return p;
}

// sin and cos of |y| <= pi / 4, and of y + q pi / 2
__device__ __forceinline__ void sincos_quadrant(double y, int q, double* sn, double* cs) {
  const double y2 = y * y;
  const double s = fma(y * y2, norm_poly(c_norm.sin_c, y2), y);
  const double c = fma(y2 * y2, norm_poly(c_norm.cos_c, y2), fma(-0.5, y2, 1.0));
  const double a = q & 1 ? c : s, b = q & 1 ? s : c;
  *sn = __hiloint2double(__double2hiint(a) ^ ((q & 2) << 30), __double2loint(a));
  *cs = __hiloint2double(__double2hiint(b) ^ (((q + 1) & 2) << 30), __double2loint(b));
}

// sin and cos of an RF phase: a two-part reduction by pi / 2 (|th| < 1e5: the
// multiple's product with the first part is exact), beyond that out of line
__device__ __forceinline__ void sincos_rf(double th, double* sn, double* cs) {
  if (!(fabs(th) < 1e5)) {
    sincos_far(th, sn, cs);
    return;
  }
  // to the nearest multiple: an addition that leaves it in the low word
  const double t = fma(th, 1.0 / (0.5 * kPi), 0x1.8p52), k = t - 0x1.8p52;
  const double y = fma(-k, c_norm.pio2_lo, fma(-k, c_norm.pio2_hi, th));
  sincos_quadrant(y, __double2loint(t), sn, cs);
}

// The RF step with cavities that load (MPBeam.cpp:2621-2704): per cavity in
// order, the ideal cavity's kick or, for an alive particle, the two
// increments of its bin from the recurrence's table (kick[((b M + j) nb +
// bin) 2 ..]); then the direct-feedback kicks of the bunch, to every
// particle.
__device__ __forceinline__ double rf_kick_dp_loading(const RingDev& r, double z, double dp,
                                                     bool alive, int j, int M, const double* zr,
                                                     const double* kick, const double* fbk) {
  int bin = -1;
  if (alive) {
    const double zmin = zr[2 * j], zmax = zr[2 * j + 1];
    const double dz = (zmax - zmin) / r.rf_bins;
    bin = (int)floor((zmax - z) / dz);
    bin = bin < 0 ? 0 : (bin >= r.rf_bins ? r.rf_bins - 1 : bin);
  }
  for (int c = 0; c < r.n_cav; ++c) {
    const int b = r.bl_index[c];
    if (b < 0) {
      double th = z * r.rf_theta_coeff[c];
      double s, co;
      sincos_rf(th, &s, &co);
      double re = fma(r.vreq_re[c], co, r.vreq_im[c] * s);
      dp = fma(re, r.inv_e_beta2, dp);
    } else if (bin >= 0) {
      const double* k = kick + (((size_t)b * M + j) * r.rf_bins + bin) * 2;
      dp += k[0];
      dp += k[1];
    }
  }
  for (int c = 0; c < r.n_cav; ++c)
    if (r.bl_index[c] >= 0 && r.bl_fb[c]) dp += fbk[(size_t)r.bl_index[c] * M + j];
  return dp;
}

// Bunch::BunchMomentumUpdateDueToRFCA (Bunch.cpp:466-472), every particle.
__device__ __forceinline__ double rf_kick_dp(const RingDev& r, double z, double dp) {
  for (int c = 0; c < r.n_cav; ++c) {
    double th = z * r.rf_theta_coeff[c];
    double s, co;
    sincos_rf(th, &s, &co);
    // Re(V e^{-i th}) = Vr cos th + Vi sin th
    double re = fma(r.vreq_re[c], co, r.vreq_im[c] * s);
    dp = fma(re, r.inv_e_beta2, dp);
  }
  return dp;
}

// Two standard normals from one Philox block: normal2 (Box-Muller on the same
// two uniforms) with
//   -2 ln u = -2 e ln 2 - 4 atanh(s), s = (m - 1) / (m + 1), u = 2^e m,
//   sqrt by a coupled Newton step on the hardware's estimate of 1 / sqrt,
//   the angle's quadrant taken from the integer before it becomes a double.
// Each within two ulps of the function.
__device__ __forceinline__ void normal2_fast(const u32x4& r, double* n0, double* n1) {
  // u = (A 2^27 + B + 1) / 2^53 in (0, 1]: the integers as the low words of
  // doubles above 2^52, the differences exact
  const double ua = __hiloint2double(0x43300000, (int)(r.v[0] >> 6));
  const double ub = __hiloint2double(0x43300000, (int)(r.v[1] >> 5));
  const double u = fma(ua, 0x1p-26, -0x1p26) + fma(ub, 0x1p-53, 0x1p-53 - 0.5);
  const int hi = __double2hiint(u);
  const int e = (hi - 0x3fe6a09e) >> 20;  // m in [sqrt(1/2), sqrt(2))
  const double m = __hiloint2double(hi - (e << 20), __double2loint(u));
  const double f = m - 1.0, d = m + 1.0;
  double rc;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(rc) : "d"(d));
  rc = fma(rc, fma(-d, rc, 1.0), rc);
  double s = f * rc;
  s = fma(rc, fma(-d, s, f), s);
  const double z = s * s;
  const double sz = s * z * norm_poly(c_norm.atanh_c, z);
  const double ed = __hiloint2double(0x43300000, e ^ (int)0x80000000) - 0x1.000008p52;  // (double)e
  // 1e-300: u = 1 gives a radius of 1e-150 in place of a division by zero
  const double t = fma(ed, c_norm.ln2_hi, 1e-300) + fma(-4.0, s, fma(ed, c_norm.ln2_lo, -4.0 * sz));
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(t));
  double g = t * y, h = 0.5 * y;
  const double er = fma(-g, h, 0.5);
  g = fma(g, er, g);
  h = fma(h, er, h);
  const double rad = fma(fma(-g, g, t), h, g);
  // angle 2 pi u2 = q pi / 2 + pi w, u2 = (A 2^27 + B) / 2^53
  const int A = (int)(r.v[2] >> 6), q = (A + (1 << 23)) >> 24;
  const double wa = __hiloint2double(0x43300000, (A - (q << 24)) ^ (int)0x80000000);
  const double wb = __hiloint2double(0x43300000, (int)(r.v[3] >> 5));
  const double w = fma(wa, 0x1p-25, -0x1.000008p27) + fma(wb, 0x1p-52, -1.0);
  double sn, cs;
  sincos_quadrant(kPi * w, q, &sn, &cs);
  *n0 = rad * cs;
  *n1 = rad * sn;
}

// Six synrad normals of particle i of bunch j at turn `turn`.
__device__ __forceinline__ void synrad_normals(uint64_t seed, uint32_t i, uint32_t j,
                                                    uint32_t turn, double (&g)[6]) {
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32) ^ kStreamSynrad;
#pragma unroll
  for (uint32_t q = 0; q < 3; ++q) {
    const u32x4 c = {{i, j, turn, q}};
    normal2_fast(philox4x32_10(c, k0, k1), &g[2 * q], &g[2 * q + 1]);
  }
}

}  // namespace cg
