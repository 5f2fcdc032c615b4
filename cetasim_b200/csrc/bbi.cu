// Broadband impedance kick (MPBeam::BBImpBeamInteraction, MPBeam.cpp:1321-1346).
//
// The reference, per bunch with charge:
//  frequency domain (MPBunch::BBImpBunchInteraction, MPBunch.cpp:2143-2346):
//    bins of width dz over [-zMax, zMax] (2n - 1 of them, n impedance
//    samples), a line-charge profile of every particle (lost ones too), a
//    Gaussian filter over the bins of one RF bucket (MPBunch.cpp:2349-2414),
//    an r2c FFT of the profile, the product with each impedance and a c2r FFT
//    back; the kick of every particle is the potential at its bin.
//  time domain (MPBunch::BBImpBunchInteractionTD, MPBunch.cpp:2029-2141):
//    bins over one RF bucket, the smoothed charge profile, per-bin mean x and
//    y of the surviving particles, and a causal sum over the bins ahead with
//    the wake table.
//
// Here the frequency-domain spectrum product is applied as what it is, a
// circular convolution of the profile with the wake sequence
// w[m] = c2r(Z)[m] / (2n - 1), computed once at set-up (k_bbi_wake_fd): the
// profile of a bunch is non-zero only on the few hundred bins its particles
// and the filter reach, so the convolution over those bins costs less than
// the two FFTs of length 2n - 1 and needs no FFT library.  The sums are the
// same up to rounding.
//
//  k_bbi_range  per-bunch lowest and highest bin and the largest |x|, |y|
//               (atomics); in the turn the longitudinal pass before it does
//               this with the positions that it writes (bbi_span_cta).
//  k_bbi_hist   per CTA: per-bin counts and sums of x and y in 64-bit fixed
//               point (the scale from the bunch's largest |x|, |y|), so the
//               result does not depend on the order of the atomics; in shared
//               memory, then added to the bunch's.
//  k_bbi_conv   one CTA per bunch: profiles, the Gaussian filter and its
//               renormalisation, the potentials of the bins that hold
//               particles; resets the accumulators.
//  k_bbi_kick   per tile: the kicks, plane by plane in the reference's order,
//               and the turn's loss check if no stage comes between.
//
// Bound by: the passes by HBM (38 MB to count, 115 MB to kick 1.6e6 particles)
// and its latency, the convolution by its chains of FMAs and barriers.  80
// bunches of 20,000, five planes, us: range 25 -> in the longitudinal pass,
// hist 53 -> 14 (global 64-bit atomics before), conv 28 -> 15 (256 threads, a
// filter with bounds checks per tap, one chain of 600 FMAs per bin and plane),
// kick 40 and the loss check 16 -> 24 together (up to fourteen divisions a
// particle).
#include <algorithm>
#include <climits>
#include <cuda_runtime.h>

#include "turn_tail.cuh"

namespace cg {

#define BBI_FULL 0xffffffffu
constexpr int kBbiThreads = 256;
// Bins up to which a CTA counts in shared memory (20 bytes each); beyond, it
// adds to the bunch's bins directly.
constexpr int kBbiSharedBins = 1024;

// Power-of-two scale of the fixed-point sums: |v| 2^s < 2^(61 - nb) for
// |v| <= amax and n < 2^nb values, so a sum of n of them stays below 2^61.
__device__ __forceinline__ int bbi_fix_exp(unsigned amax_hi, int n) {
  const double a = __hiloint2double((int)amax_hi, 0);
  if (!(a > 0) || isinf(a)) return 0;
  const int nb = 32 - __clz(n);
  return 60 - ilogb(a) - nb;
}

__global__ void __launch_bounds__(kTile) k_bbi_range(const double* __restrict__ c, int64_t npad,
                                                     const uint8_t* __restrict__ surv,
                                                     const int* __restrict__ tile_bunch,
                                                     const BunchDev* __restrict__ bunch,
                                                     const __grid_constant__ BbiParams p,
                                                     BbiSpan* span, int* status) {
  const int b = tile_bunch[blockIdx.x];
  const BunchDev& Bd = bunch[b];
  const int64_t g = (int64_t)blockIdx.x * kTile + threadIdx.x;
  const bool valid = (blockIdx.x - Bd.tile_off) * kTile + (int)threadIdx.x < Bd.n;
  bbi_span_cta(p, span + b, status, valid && Bd.q_macro != 0, valid && surv[g] == kAlive,
               valid ? c[g] : 0.0, valid ? c[2 * npad + g] : 0.0, valid ? c[4 * npad + g] : 0.0);
}

__global__ void __launch_bounds__(kBbiThreads) k_bbi_hist(const double* __restrict__ c, int64_t npad,
                                                          const uint8_t* __restrict__ surv,
                                                          const BunchDev* __restrict__ bunch,
                                                          int tiles,
                                                          const __grid_constant__ BbiParams p,
                                                          const BbiSpan* __restrict__ span,
                                                          int* status, int* cnt,
                                                          unsigned long long* sxy) {
  extern __shared__ unsigned s_bin[];  // W counts, then x (lo, hi), y (lo, hi)
  const int b = blockIdx.x, t0 = blockIdx.y * tiles;
  const BunchDev& Bd = bunch[b];
  if (Bd.q_macro == 0 || t0 >= Bd.n_tiles) return;
  const BbiSpan S = span[b];
  const int first = S.lo(), W = S.bins();
  if (W < 1) return;
  if (W > CG_BBI_MAX_BINS) {
    if (threadIdx.x == 0) atomicOr(status, kStatusBbiWide);
    return;
  }
  const bool shared = W <= kBbiSharedBins;
  if (shared) {
    for (int t = threadIdx.x; t < 5 * W; t += kBbiThreads) s_bin[t] = 0u;
    __syncthreads();
  }
  const Pow2 fx = pow2_split(bbi_fix_exp(S.ax, Bd.n));
  const Pow2 fy = pow2_split(bbi_fix_exp(S.ay, Bd.n));
  const size_t base = (size_t)b * p.wcap;
  int64_t g = (int64_t)(Bd.tile_off + t0) * kTile + threadIdx.x;
  int i = t0 * kTile + threadIdx.x;
  for (int u = 0; u < tiles && i < Bd.n; ++u, g += kTile, i += kTile) {
    const double x = c[g], y = c[2 * npad + g];
    const int idx = bbi_bin(p, c[4 * npad + g]);
    const bool sums = !p.td || surv[g] == kAlive;
    if (idx < 0) continue;
    const int t = idx - first;
    if (shared) atomicAdd(&s_bin[t], 1u);
    else atomicAdd(&cnt[base + t], 1);
    if (!sums) continue;
    const long long qx = __double2ll_rn(pow2_scale(x, fx)), qy = __double2ll_rn(pow2_scale(y, fy));
    if (shared) {
      add64_split(&s_bin[W + t], &s_bin[2 * W + t], qx);
      add64_split(&s_bin[3 * W + t], &s_bin[4 * W + t], qy);
    } else {
      atomicAdd(&sxy[2 * base + t], (unsigned long long)qx);  // two's complement sums
      atomicAdd(&sxy[2 * base + p.wcap + t], (unsigned long long)qy);
    }
  }
  if (!shared) return;
  __syncthreads();
  for (int t = threadIdx.x; t < W; t += kBbiThreads) {
    if (!s_bin[t]) continue;
    atomicAdd(&cnt[base + t], (int)s_bin[t]);
    atomicAdd(&sxy[2 * base + t], (unsigned long long)s_bin[2 * W + t] << 32 | s_bin[W + t]);
    atomicAdd(&sxy[2 * base + p.wcap + t],
              (unsigned long long)s_bin[4 * W + t] << 32 | s_bin[3 * W + t]);
  }
}

// One CTA per bunch.  pot[(b * 6 + q) * wcap + t] for the bins a + t:
// q = 0 the smoothed charge profile; q = 1..5 the potentials of the planes
// Z, Dx, Dy, Qx, Qy at the bins that hold particles (frequency domain: the
// wakePotenFromBBI arrays, MPBunch.cpp:2193-2341; time domain: temp[0..4],
// MPBunch.cpp:2100-2111), 0 at the other bins.
//
// Three profiles side by side (the charge, the dipoles x and y; time domain:
// the charge and the mean x and y, which are not smoothed), the tasks
// (profile, bin) and (plane, bin) over the threads; a sum over bins runs in
// four chains.  Smoothing is GetSmoothedBunchProfileGassionFilter
// (MPBunch.cpp:2349-2414): the K = 51 Gaussian filter with end-value padding
// over the bins [s0, s1), then the filtered profile scaled so that its sum
// over [s0, s1) equals the raw one; bins outside pass unchanged, every other
// bin of the profile is zero and stays zero.  The raw profiles keep kBbiHalf
// zeros on both sides, so that a tap away from s0 and s1 needs no check.
template <int NT>
__global__ void __launch_bounds__(NT, 1) k_bbi_conv(
    const BunchDev* __restrict__ bunch, const __grid_constant__ BbiParams p,
    const double* __restrict__ w, BbiSpan* span, int* cnt,
    unsigned long long* sxy, double* pot, int2* win) {
  extern __shared__ double sm[];
  __shared__ double red[NT / 32][6];
  __shared__ double scale[3];
  const int b = blockIdx.x;
  const BunchDev& Bd = bunch[b];
  const BbiSpan S = span[b];
  const int W = S.bins(), l = S.lo(), h = l + W - 1;
  if (Bd.q_macro == 0 || W < 1 || W > CG_BBI_MAX_BINS) {
    if (threadIdx.x == 0) {
      win[b] = make_int2(0, 0);
      span[b] = BbiSpan{0u, 0u, 0u, 0u};
    }
    return;
  }
  const int a = max(l - kBbiHalf, 0);
  const int e = min(h + kBbiHalf, p.nbins - 1);
  const int n = e - a + 1;
  const int nr = n + 2 * kBbiHalf;    // raw bins a - kBbiHalf ..
  double* s_raw = sm;                 // 3 x nr
  double* s_p = sm + 3 * (size_t)nr;  // 3 x n
  const size_t base = (size_t)b * p.wcap;
  const int ex = bbi_fix_exp(S.ax, Bd.n), ey = bbi_fix_exp(S.ay, Bd.n);
  // the charge per bin: frequency domain a line charge [C/s]
  // (macroEleCharge e / dz c, MPBunch.cpp:2172), time domain [C] (:2054)
  const double unit = p.td ? Bd.q_macro * kElectronCharge
                           : Bd.q_macro * kElectronCharge / p.dz * kCLight;
  const int smooth = p.td ? 1 : 3;  // profiles that are smoothed
  for (int t = threadIdx.x; t < nr; t += NT) {
    const int j = a - kBbiHalf + t - l;
    double r0 = 0, r1 = 0, r2 = 0;
    if (j >= 0 && j < W) {
      const int n0 = cnt[base + j];
      r0 = n0 * unit;
      const double sx = scalbn((double)(long long)sxy[2 * base + j], -ex);
      const double sy = scalbn((double)(long long)sxy[2 * base + p.wcap + j], -ey);
      if (!p.td) {  // the dipole profiles (MPBunch.cpp:2261-2273, 2304-2316)
        r1 = unit * sx;
        r2 = unit * sy;
      } else if (n0 > 0) {
        // mean x, y of the survivors over all the bin's particles (MPBunch.cpp:2061-2082)
        r1 = sx / n0;
        r2 = sy / n0;
      }
      // leave the accumulators zero for the next call
      cnt[base + j] = 0;
      sxy[2 * base + j] = 0ull;
      sxy[2 * base + p.wcap + j] = 0ull;
    }
    s_raw[t] = r0;
    s_raw[nr + t] = r1;
    s_raw[2 * nr + t] = r2;
  }
  __syncthreads();
  double sum[6] = {0, 0, 0, 0, 0, 0};  // raw and filtered sums of the profiles
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const double* raw = s_raw + q * nr + kBbiHalf;
    // the profiles one after the other over the threads
    for (int t = ((int)threadIdx.x + NT - q * n % NT) % NT;
         t < n; t += NT) {
      const int i = a + t;
      double y = raw[t];
      if (q < smooth && i >= p.s0 && i < p.s1) {
        if (i - kBbiHalf >= p.s0 && i + kBbiHalf < p.s1) {
          double y0 = p.g[0] * raw[t - kBbiHalf], y1 = 0, y2 = 0;
#pragma unroll
          for (int k = 1; k <= 2 * kBbiHalf; k += 2) {
            y1 = fma(p.g[k], raw[t + k - kBbiHalf], y1);
            y2 = fma(p.g[k + 1], raw[t + k + 1 - kBbiHalf], y2);
          }
          y = y0 + (y1 + y2);
        } else {
          y = 0;
          for (int k = -kBbiHalf; k <= kBbiHalf; ++k) {
            int jj = i + k;
            jj = jj < p.s0 ? p.s0 : (jj >= p.s1 ? p.s1 - 1 : jj);  // end-value padding
            y = fma(p.g[k + kBbiHalf], jj >= a && jj <= e ? raw[jj - a] : 0.0, y);
          }
        }
        sum[2 * q] += raw[t];
        sum[2 * q + 1] += y;
      }
      s_p[q * n + t] = y;
    }
  }
#pragma unroll
  for (int q = 0; q < 6; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum[q] += __shfl_xor_sync(BBI_FULL, sum[q], o);
  }
  if ((threadIdx.x & 31) == 0)
    for (int q = 0; q < 6; ++q) red[threadIdx.x >> 5][q] = sum[q];
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      double v = threadIdx.x < NT / 32 ? red[threadIdx.x][q] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(BBI_FULL, v, o);
      sum[q] = v;
    }
    // MPBunch.cpp:2404-2407 (0 / 0 when empty, as there)
    if (threadIdx.x < 3) {
      const double s0 = threadIdx.x == 0 ? sum[0] : threadIdx.x == 1 ? sum[2] : sum[4];
      const double s1 = threadIdx.x == 0 ? sum[1] : threadIdx.x == 1 ? sum[3] : sum[5];
      scale[threadIdx.x] = s0 / s1;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < smooth * n; t += NT) {
    const int q = t >= 2 * n ? 2 : t >= n ? 1 : 0, i = a + t - q * n;
    if (i >= p.s0 && i < p.s1) s_p[t] *= scale[q];
  }
  __syncthreads();
  double* out = pot + (size_t)b * 6 * p.wcap;
  for (int t = threadIdx.x; t < n; t += NT) out[t] = s_p[t];
  const int N = p.nbins;
  for (int task = threadIdx.x; task < 5 * n; task += NT) {
    const int q = task / n, t = task - q * n, i = a + t;
    double v = 0;
    if (i >= l && i <= h && p.sim[q]) {
      const double* wq = w + (size_t)q * p.nw;
      double s[4] = {0, 0, 0, 0};
      if (!p.td) {
        // V_q(i) = sum_j P(j) w_q((i - j) mod N): the c2r of the profile's
        // spectrum times Z_q, over N (MPBunch.cpp:2193-2198 and after)
        const double* P = s_p + (q == 1 ? n : q == 2 ? 2 * n : 0);
        int u = 0;
        for (; u + 4 <= n; u += 4)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int m = t - u - k;
            s[k] = fma(P[u + k], __ldg(wq + (m < 0 ? m + N : m)), s[k]);
          }
        for (; u < n; ++u) s[0] = fma(P[u], __ldg(wq + (t - u < 0 ? t - u + N : t - u)), s[0]);
        v = (s[0] + s[1]) + (s[2] + s[3]);
        if (q == 0) v = -v;  // wakePotenZ = -temp / nBins (MPBunch.cpp:2198)
      } else {
        // the bins ahead, j = i .. (MPBunch.cpp:2102-2111), wake sample j - i
        const double* P = s_p + t;
        const double* D = q == 1 ? s_p + n + t : q == 2 ? s_p + 2 * n + t : nullptr;
        const int m = min(e, i + p.nw - 1) - i + 1;
        int u = 0;
        for (; u + 4 <= m; u += 4)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const double f = __ldg(wq + u + k) * P[u + k];
            s[k] = D ? fma(-f, D[u + k], s[k]) : s[k] - f;
          }
        for (; u < m; ++u) {
          const double f = __ldg(wq + u) * P[u];
          s[0] = D ? fma(-f, D[u], s[0]) : s[0] - f;
        }
        v = (s[0] + s[1]) + (s[2] + s[3]);
      }
    }
    out[(size_t)(1 + q) * p.wcap + t] = v;
  }
  if (threadIdx.x == 0) {
    win[b] = make_int2(a, n);
    span[b] = BbiSpan{0u, 0u, 0u, 0u};
  }
}

// The kicks (frequency domain MPBunch.cpp:2201-2342, time domain
// MPBunch.cpp:2113-2121), the planes in the reference's order: a potential
// over E beta^2 and, transversely, the beta function.
struct BbiScale {
  double z, x, y;
};
template <bool MARK>
__global__ void __launch_bounds__(kTile) k_bbi_kick(double* __restrict__ c, int64_t npad,
                                                    uint8_t* __restrict__ surv,
                                                    const int* __restrict__ tile_bunch,
                                                    const BunchDev* __restrict__ bunch,
                                                    const __grid_constant__ BbiParams p,
                                                    const int2* __restrict__ win,
                                                    const double* __restrict__ pot,
                                                    const __grid_constant__ BbiScale f,
                                                    const __grid_constant__ Aperture ap,
                                                    int* loss_count) {
  const int b = tile_bunch[blockIdx.x];
  const BunchDev& Bd = bunch[b];
  const int64_t g = (int64_t)blockIdx.x * kTile + threadIdx.x;
  const bool valid = (blockIdx.x - Bd.tile_off) * kTile + (int)threadIdx.x < Bd.n;
  double x = 0, y = 0, z = 0;
  if (valid) {
    x = c[g];
    y = c[2 * npad + g];
    z = c[4 * npad + g];
  }
  const int2 wn = win[b];
  const int idx = valid && Bd.q_macro != 0 && wn.y != 0 ? bbi_bin(p, z) : -1;
  if (idx >= 0) {
    double px = c[npad + g], py = c[3 * npad + g], dp = c[5 * npad + g];
    const double* v = pot + (size_t)b * 6 * p.wcap + (idx - wn.x);
    const double z0 = f.z * v[p.wcap], dx = f.x * v[2 * p.wcap], dy = f.y * v[3 * p.wcap];
    const double qx = f.x * v[4 * p.wcap], qy = f.y * v[5 * p.wcap];
    if (p.sim[0]) dp += z0;
    if (!p.td) {
      if (p.sim[3]) px = fma(qx, x, px);
      if (p.sim[4]) py = fma(qy, y, py);
      if (p.sim[1]) px += dx;
      if (p.sim[2]) py += dy;
    } else {
      if (p.sim[1]) px += dx;
      if (p.sim[2]) py += dy;
      if (p.sim[3]) px = fma(qx, x, px);
      if (p.sim[4]) py = fma(qy, y, py);
    }
    c[npad + g] = px;
    c[3 * npad + g] = py;
    c[5 * npad + g] = dp;
  }
  if (MARK) mark_lost_warp(ap, valid, x, y, z, surv + g, loss_count + b);
}

size_t bbi_span_bytes() { return sizeof(BbiSpan); }

cudaError_t launch_bbi(Handle& h, bool have_range, bool mark) {
  const BbiParams& p = h.bbi;
  BbiSpan* span = reinterpret_cast<BbiSpan*>(h.d.bbi_span);
  const double fz = 1.0 / p.energy / p.beta2;
  const BbiScale f = {fz, fz / p.beta_x, fz / p.beta_y};
  if (!have_range)
    k_bbi_range<<<h.n_tiles, kTile, 0, h.stream>>>(h.d.c, h.npad, h.d.surv, h.d.tile_bunch,
                                                   h.d.bunch, p, span, h.d.status);
  // six CTAs per SM: each ends with an atomic per bin and sum, so no more CTAs
  // than the particles' reads need (two tiles each: 20 us, eight: 13.7)
  int big = 1;
  for (int j = 0; j < h.M; ++j) big = std::max(big, h.tile_off[j + 1] - h.tile_off[j]);
  const int tiles = std::max(1, (h.n_tiles + 148 * 6 - 1) / (148 * 6));
  k_bbi_hist<<<dim3(h.M, (big + tiles - 1) / tiles), kBbiThreads,
               5 * sizeof(unsigned) * std::min(p.wcap, kBbiSharedBins), h.stream>>>(
      h.d.c, h.npad, h.d.surv, h.d.bunch, tiles, p, span, h.d.status, h.d.bbi_cnt, h.d.bbi_sxy);
  // a bunch's few thousand tasks want 1024 threads where each SM has a bunch or
  // less; beyond, several CTAs of 256 share an SM
  // (900 bunches of 270 particles, a kick 92 -> 75 us; 900 of 4000, a turn with the
  // wake table 304 -> 285 us)
  const bool few = h.M <= 148;
  (few ? k_bbi_conv<1024> : k_bbi_conv<256>)<<<h.M, few ? 1024 : 256, bbi_conv_smem(p), h.stream>>>(
      h.d.bunch, p, h.d.bbi_w, span, h.d.bbi_cnt, h.d.bbi_sxy, h.d.bbi_pot, h.d.bbi_win);
  (mark ? k_bbi_kick<true> : k_bbi_kick<false>)<<<h.n_tiles, kTile, 0, h.stream>>>(
      h.d.c, h.npad, h.d.surv, h.d.tile_bunch, h.d.bunch, p, h.d.bbi_win, h.d.bbi_pot, f, aperture(h),
      h.d.loss_count);
  return cudaGetLastError();
}

size_t bbi_conv_smem(const BbiParams& p) {
  return (size_t)(6 * p.wcap + 6 * kBbiHalf) * sizeof(double);
}

cudaError_t prepare_bbi(const BbiParams& p) {
  cudaError_t e = cudaFuncSetAttribute(k_bbi_conv<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)bbi_conv_smem(p));
  return e != cudaSuccess ? e : cudaFuncSetAttribute(k_bbi_conv<256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     (int)bbi_conv_smem(p));
}

// ---------------------------------------------------------------------------
// Set-up of the frequency-domain wake sequences: w_q[m] = c2r(X_q)[m] / N with
// N = 2n - 1 and X_q the impedance of plane q (times i for the transverse
// planes, MPBunch.cpp:2212 and after): for odd N, c2r takes X_0's real part
// and the Hermitian extension of X_1 .. X_{n-1}, so
//   w[m] = (Re X_0 + 2 sum_{k=1}^{n-1} Re(X_k e^{2 pi i k m / N})) / N.
// Twiddles come from a table indexed by (k m) mod N.

__global__ void k_bbi_twiddle(double2* tw, int N) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= N) return;
  double s, c;
  sincospi(2.0 * (double)r / (double)N, &s, &c);
  tw[r] = make_double2(c, s);
}

__global__ void k_bbi_wake_fd(const double2* __restrict__ X, const double2* __restrict__ tw, int n,
                              int N, double* w) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  const int q = blockIdx.y;
  if (m >= N) return;
  const double2* Xq = X + (size_t)q * n;
  double s = 0;
  int r = 0;  // (k m) mod N
  for (int k = 1; k < n; ++k) {
    r += m;
    if (r >= N) r -= N;
    const double2 t = tw[r];
    s = fma(Xq[k].x, t.x, fma(-Xq[k].y, t.y, s));
  }
  w[(size_t)q * N + m] = (Xq[0].x + 2.0 * s) / N;
}

cudaError_t bbi_wake_fd(const double2* d_X, int n, double* d_w, cudaStream_t st) {
  const int N = 2 * n - 1;
  double2* tw = nullptr;
  cudaError_t e = cudaMallocAsync(&tw, sizeof(double2) * N, st);
  if (e != cudaSuccess) return e;
  k_bbi_twiddle<<<(N + 255) / 256, 256, 0, st>>>(tw, N);
  k_bbi_wake_fd<<<dim3((N + 127) / 128, 5), 128, 0, st>>>(d_X, tw, n, N, d_w);
  e = cudaGetLastError();
  cudaError_t f = cudaFreeAsync(tw, st);
  return e != cudaSuccess ? e : f;
}

}  // namespace cg
