// Device pieces that the broadband impedance and the longitudinal pass share:
// the bin of a particle, the bunches' ranges, and the loss check.
#pragma once
#include <climits>

#include "kernels.cuh"
#include "track_math.cuh"

namespace cg {

// What a kick collects of a bunch first, as maxima over its particles that are
// zero without any and between kicks: its highest and lowest bin and the high
// words of its largest |x| and |y|; in a cache line of its own (the lines of
// all bunches behind one L2 slice would queue the atomics of all CTAs).
struct alignas(128) BbiSpan {
  unsigned top, bottom;  // highest bin + 1, INT_MAX - lowest bin
  unsigned ax, ay;
  __device__ __forceinline__ int lo() const { return INT_MAX - (int)bottom; }
  __device__ __forceinline__ int bins() const { return top ? (int)top - lo() : 0; }
};

// s / d correctly rounded from inv = 1 / d, for bins whose edges the quotient
// decides: the product is within two units in the last place, the first
// correction leaves less than one, and the second then rounds as the division
// does (P. W. Markstein, IBM J. Res. Dev. 34 (1990) 111: a residual exact by
// FMA, times a correctly rounded reciprocal).  A division costs the kernels of
// the space charge 9 % of their turn, the branch on its slow path above all.
__device__ __forceinline__ double bin_quotient(double s, double d, double inv) {
  double q = s * inv;
  q = fma(fma(-q, d, s), inv, q);
  return fma(fma(-q, d, s), inv, q);
}

// The bin of a particle, or -1 when the reference would index outside its
// profile.  Frequency domain (z - zMin + dz / 2) / dz (MPBunch.cpp:2170),
// time domain (z - zMin) / dz (MPBunch.cpp:2052), truncated as int() does
// (so -1 < t < 0 is bin 0).  The product with 1 / dz, within 2^-51 of the quotient
// (relative), decides unless a whole number lies within 2^-50, where the division
// is taken: next to the longitudinal pass that costs less than bin_quotient
// (impedance_spectrum 500 us, 507).
__device__ __forceinline__ int bbi_bin(const BbiParams& p, double z) {
  const double s = p.td ? z - p.zmin : (z - p.zmin) + p.dz / 2;
  double t = s * p.inv_dz;
  const double whole = (t + 0x1.8p52) - 0x1.8p52;
  if (!(fabs(t - whole) > 0x1p-50 * fabs(t))) t = s / p.dz;
  return (t > -1.0 && t < (double)p.nbins) ? (int)t : -1;
}

// A CTA's particles into their bunch's span; every thread of the CTA calls it.
// Frequency domain: every particle enters the dipole profiles (MPBunch.cpp:
// 2265-2270); time domain: the survivors' means (:2061-2070).  Of the largest
// |x|, |y| only the exponent is used (the scale of the fixed-point sums).
__device__ __forceinline__ void bbi_span_cta(const BbiParams& p, BbiSpan* span, int* status,
                                             bool valid, bool alive, double x, double y, double z) {
  __shared__ unsigned s_max[4];
  if (threadIdx.x < 4) s_max[threadIdx.x] = 0u;
  __syncthreads();
  const int idx = valid ? bbi_bin(p, z) : -1;
  if (valid && idx < 0) atomicOr(status, kStatusBbiRange);
  if (__any_sync(0xffffffffu, idx >= 0)) {
    const bool in = idx >= 0 && (!p.td || alive);
    // a NaN is not a maximum
    const unsigned ax = in ? (unsigned)__double2hiint(fmax(fabs(x), 0.0)) : 0u;
    const unsigned ay = in ? (unsigned)__double2hiint(fmax(fabs(y), 0.0)) : 0u;
    const unsigned m[4] = {__reduce_max_sync(0xffffffffu, (unsigned)(idx + 1)),
                           __reduce_max_sync(0xffffffffu, idx < 0 ? 0u : (unsigned)(INT_MAX - idx)),
                           __reduce_max_sync(0xffffffffu, ax), __reduce_max_sync(0xffffffffu, ay)};
    if ((threadIdx.x & 31) == 0)
#pragma unroll
      for (int q = 0; q < 4; ++q) atomicMax(&s_max[q], m[q]);
  }
  __syncthreads();
  if (threadIdx.x < 4 && s_max[threadIdx.x]) atomicMax(&span->top + threadIdx.x, s_max[threadIdx.x]);
}

// The same for the short-range wake: the survivors' range of z, as maxima of
// ordered keys (of z and of -z).
struct alignas(128) SrSpan {
  unsigned long long top, bottom;
};
struct SrDev {
  SrSpan* span;
  int* counts;         // M x B particles per bin
  double *sumx, *sumy; // M x B
  int B;
};
// doubles as unsigned integers of the same order, none of them zero
__device__ __forceinline__ unsigned long long sr_key(double z) {
  const long long b = __double_as_longlong(z);
  return b < 0 ? ~(unsigned long long)b : (unsigned long long)b | 1ull << 63;
}
__device__ __forceinline__ double sr_unkey(unsigned long long k) {
  return __longlong_as_double((long long)(k >> 63 ? k & ~(1ull << 63) : ~k));
}
// A CTA's particles into their bunch's span; every thread of the CTA calls it.
// The CTA of the bunch's first tile clears the counts of the call before.
__device__ __forceinline__ void sr_span_cta(const SrDev& sr, int b, bool first, bool alive, double z) {
  __shared__ unsigned long long s_key[2];
  if (threadIdx.x < 2) s_key[threadIdx.x] = 0ull;
  if (first)
    for (int q = threadIdx.x; q < sr.B; q += blockDim.x) {
      sr.counts[(size_t)b * sr.B + q] = 0;
      sr.sumx[(size_t)b * sr.B + q] = sr.sumy[(size_t)b * sr.B + q] = 0.0;
    }
  __syncthreads();
  // the extremes without NaN, as fmin and fmax leave it out
  double mx = alive ? z : NAN, mn = mx;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  }
  if ((threadIdx.x & 31) == 0 && mx == mx) {
    atomicMax(&s_key[0], sr_key(mx));
    atomicMax(&s_key[1], sr_key(-mn));
  }
  __syncthreads();
  if (threadIdx.x < 2 && s_key[threadIdx.x]) atomicMax(&sr.span[b].top + threadIdx.x, s_key[threadIdx.x]);
}

SrDev sr_dev(const Handle& h);

// Bunch::MarkLostParticle (Bunch.cpp:172-200) for the warp's particles, their
// number of loss conditions added to the bunch's.  A position clearly inside
// the aperture by the reciprocals takes no division; the others take the
// reference's.
struct Aperture {
  double ax, ay, iax, iay, z_loss;
};
__device__ __forceinline__ void mark_lost_warp(const Aperture& ap, bool valid, double x, double y,
                                               double z, uint8_t* surv, int* loss_count) {
  const double tx = x * ap.iax, ty = y * ap.iay;
  int count = 0;
  if (valid && !(fma(tx, tx, ty * ty) < 0.999 && fabs(z) <= ap.z_loss)) {
    uint8_t s = *surv;
    count = mark_lost_particle(ap.z_loss, ap.ax, ap.ay, x, y, z, &s);
    if (count) *surv = s;
  }
  if (__any_sync(0xffffffffu, count)) {
    count = __reduce_add_sync(0xffffffffu, count);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss_count, count);
  }
}

Aperture aperture(const Handle& h);

// 2^e in two factors (one can be beyond a double's range), and v 2^e: exact as
// scalbn, in two products instead of its thirty instructions.
struct Pow2 {
  double a, b;
};
__device__ __forceinline__ Pow2 pow2_split(int e) {
  const int h = e >> 1;
  return {__hiloint2double((1023 + h) << 20, 0), __hiloint2double((1023 + e - h) << 20, 0)};
}
__device__ __forceinline__ double pow2_scale(double v, const Pow2& f) { return v * f.a * f.b; }

// A 64-bit sum in shared memory as two words (a 64-bit shared atomic is a
// compare-and-swap loop, which retries under contention; the carry of a 32-bit
// add is exact).
__device__ __forceinline__ void add64_split(unsigned* lo, unsigned* hi, long long v) {
  const unsigned vl = (unsigned)v, old = atomicAdd(lo, vl);
  const unsigned vh = (unsigned)((unsigned long long)v >> 32) + (old + vl < vl ? 1u : 0u);
  if (vh) atomicAdd(hi, vh);
}

}  // namespace cg
