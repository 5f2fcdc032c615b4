// Short-range wake (MPBunch::BunchTransferDueToSRWake, MPBunch.cpp:1887-2025).
//
//  k_sr_range per-bunch range of z over the survivors (GetZMinMax,
//             MPBunch.cpp:1860-1884), and the last call's counts cleared; in
//             the turn the longitudinal pass before it does this with the
//             positions that it writes (sr_span_cta).
//  k_sr_bins  two independent jobs in one launch.  Histogram CTAs: the
//             bunch's bins [zMin - 2 sigma_z, zMax + 2 sigma_z] (the last rms
//             bunch length) filled in shared memory with warp-aggregated
//             atomics (__match_any_sync groups lanes hitting the same bin),
//             integer counts so the result is exact and order-independent,
//             and for the transverse potentials the per-bin sums of x and y
//             over alive particles.  Lag CTAs: below.
//             The 1 mm pseudo-Green wake W_z at the 2B-1 distinct lags
//             tau = (i - j) dtBin (WakeFunction.cpp:558-653).  The reference
//             evaluates it for all B^2 bin pairs; the lag set is identical.
//             The 1000-term sum per resonator splits over a CTA; the
//             lag-independent cos/sin factors are tabulated once at setup.
//  k_sr_pot   V_i = (V_i(previous turn) + sum_j W(i - j) n_j) (-e q/E)
//             (the reference keeps srWakePoten between turns,
//             MPBunch.cpp:1894-1897, and only the longitudinal plane kicks).
//             A warp per bin, its lanes over j.
//  k_sr_kick  dp += V[bin] for alive particles, and the turn's loss check if
//             no stage comes between.
//
// Bound by latency for a single bunch (five dependent launches of a few
// thousand cycles), by HBM for a train.  One bunch of 1e5 particles, 100 bins,
// us: range 44 (one thread over the tiles) -> in the longitudinal pass,
// histogram and lags 8 + 5 -> 6.4 together, potentials 7 -> 4.1 (a thread per
// bin before), kick and loss check 5 + 7 -> 5.0 together.
#include <algorithm>
#include <cuda_runtime.h>
#include "turn_tail.cuh"

namespace cg {

#define FULL_MASK 0xffffffffu

constexpr int kSrGreenN = 1000;  // nz of GetBBRPusdoWakeFun

struct SrResonator {
  double dz;       // zMax / nz
  double c;        // 2 Q / vz
  double coeff;    // sqrt(2/pi) Rs c / sigma_z
};

__device__ __forceinline__ double warp_sum1(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
  return v;
}

__global__ void __launch_bounds__(kTile) k_sr_range(const double* __restrict__ c, int64_t npad,
                                                    const uint8_t* __restrict__ surv,
                                                    const int* __restrict__ tile_bunch,
                                                    const BunchDev* __restrict__ bunch, SrDev sr) {
  const int b = tile_bunch[blockIdx.x];
  const BunchDev& Bd = bunch[b];
  const int64_t g = (int64_t)blockIdx.x * kTile + threadIdx.x;
  const bool valid = (blockIdx.x - Bd.tile_off) * kTile + (int)threadIdx.x < Bd.n;
  sr_span_cta(sr, b, (int)blockIdx.x == Bd.tile_off, valid && surv[g] == kAlive,
              valid ? c[4 * npad + g] : 0.0);
}

// A bunch's bins (GetZMinMax seeds both extremes with particle 0, alive or not).
struct SrGeom {
  double lo, dz;
};
__device__ __forceinline__ SrGeom sr_geometry(const SrSpan& s, double z0, double bunch_length, int B) {
  double zmin = z0, zmax = z0;
  if (s.top) {
    zmin = fmin(zmin, -sr_unkey(s.bottom));
    zmax = fmax(zmax, sr_unkey(s.top));
  }
  zmin = zmin - 1.e-6;
  zmax = zmax + 1.e-6;
  const double lo = zmin - 2 * bunch_length, hi = zmax + 2 * bunch_length;
  return {lo, (hi - lo) / B};
}

// truncation toward zero, as int() in the reference; inv = 1 / dz
__device__ __forceinline__ int sr_bin(double z, double lo, double dz, double inv, int B) {
  const double t = bin_quotient(z - lo, dz, inv);
  return (t > -1.0 && t < (double)B) ? (int)t : -1;
}

// One chunk of particles into its bunch's bins.  XY: the sums of x and y too.
template <bool XY>
__device__ __forceinline__ void sr_hist_chunk(const double* __restrict__ c, int64_t npad,
                                              const uint8_t* __restrict__ surv, const int4& l, int n,
                                              int tile_off, const SrGeom& G, int* counts,
                                              double* sumx, double* sumy, int B,
                                              unsigned char* sm_raw) {
  int* s_cnt = reinterpret_cast<int*>(sm_raw);
  double* s_x = reinterpret_cast<double*>(sm_raw + ((B * sizeof(int) + 15) & ~(size_t)15));
  double* s_y = s_x + B;
  for (int q = threadIdx.x; q < B; q += kTile) {
    s_cnt[q] = 0;
    if (XY) s_x[q] = s_y[q] = 0.0;
  }
  __syncthreads();
  const double inv = 1.0 / G.dz;
  int64_t g = (int64_t)l.y * kTile + threadIdx.x;
  int i = (l.y - tile_off) * kTile + threadIdx.x;
  for (int u = 0; u < l.z; ++u, g += kTile, i += kTile) {
    const int idx = i < n ? sr_bin(c[4 * npad + g], G.lo, G.dz, inv, B) : -1;
    // warp-aggregated count: one shared atomic per distinct bin in the warp
    const unsigned peers = __match_any_sync(FULL_MASK, idx);
    if (idx >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&s_cnt[idx], __popc(peers));
    if (XY && idx >= 0 && surv[g] == kAlive) {
      atomicAdd(&s_x[idx], c[g]);
      atomicAdd(&s_y[idx], c[2 * npad + g]);
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < B; q += kTile) {
    if (!s_cnt[q]) continue;
    atomicAdd(&counts[q], s_cnt[q]);
    if (XY) {
      atomicAdd(&sumx[q], s_x[q]);
      atomicAdd(&sumy[q], s_y[q]);
    }
  }
}

// e^{-x} I_nu(x) for nu = 1/4, 5/4, 3/4, 7/4 (in that order), over the 256
// threads of the CTA: the power series sum_k (x/2)^{2k+nu} / (k! Gamma(k+nu+1)),
// each term formed in logarithms (so e^{-x} and the peak near k = x/2 stay in
// range) and summed up to 12 standard widths past the peak.  Thread 0 gets
// the four sums.
__device__ void scaled_bessel_i4(double x, double (&out)[4], double (*sw4)[8]) {
  const double nu[4] = {0.25, 1.25, 0.75, 1.75};
  const int K = (int)(0.5 * x + 12.0 * sqrt(0.5 * x + 1.0) + 40.0);
  const double lx = log(0.5 * x);
  double s[4] = {0, 0, 0, 0};
  for (int k = threadIdx.x; k <= K; k += blockDim.x) {
    const double lk = lgamma(k + 1.0);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      s[q] += exp((2 * k + nu[q]) * lx - lk - lgamma(k + nu[q] + 1.0) - x);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const double v = warp_sum1(s[q]);
    if ((threadIdx.x & 31) == 0) sw4[q][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int q = 0; q < 4; ++q) {
      double a = 0.0;
      for (int w = 0; w < 8; ++w) a += sw4[q][w];
      out[q] = a;
    }
  __syncthreads();
}

// GetRWPusdoWakeFun's longitudinal function fu_z(u) (WakeFunction.cpp:
// 387-444), zero outside 1e-2 <= |u| <= 40; valid in thread 0.
__device__ double rw_pseudo_fz(double u, double (*sw4)[8]) {
  if (fabs(u) < 1.e-2 || fabs(u) > 40) return 0.0;
  const double x = u * u / 4.0;
  double bi[4];
  scaled_bessel_i4(x, bi, sw4);
  // I_{-3/4} = (2 (1/4) / x) I_{1/4} + I_{5/4};  I_{-1/4} = (2 (3/4) / x) I_{3/4} + I_{7/4}
  const double p025 = bi[0], m075 = 2.0 * 0.25 / x * bi[0] + bi[1];
  const double p075 = bi[2], m025 = 2.0 * 0.75 / x * bi[2] + bi[3];
  const double c1 = pow(fabs(u), 1.5);  // times e^{-x}, already in the scaled sums
  const double c2 = u > 0 ? 1 : -1;
  return c1 * (c2 * (m025 - p075) + (-p025 + m075));
}

// A CTA: W_z(tau) summed over resonators, lag bin m = i - j of bunch b.
__device__ __forceinline__ void sr_lag_cta(int b, int m, double dz, const SrResonator* __restrict__ res,
                                           const double* __restrict__ green, int n_res, int B,
                                           double sigmat, double rw_coeff, double* lag,
                                           const double* __restrict__ green_t) {
  __shared__ double sw[8];
  __shared__ double sw4[4][8];
  const double dtBin = dz / kCLight;
  const double tau = m * dtBin;
  const double u = tau / sigmat;
  double total = 0.0;
  // resistive-wall sectors (GetRWSRWakeFun, WakeFunction.cpp:446-497; the
  // reference adds them before the resonators, MPBunch.cpp:1968-1978)
  if (rw_coeff != 0.0) {
    const double fz = rw_pseudo_fz(u, sw4);
    if (threadIdx.x == 0) total += rw_coeff * fz;
  }
  for (int r = 0; r < n_res; ++r) {
    const SrResonator R = res[r];
    double s = 0.0;
    for (int j = threadIdx.x; j < kSrGreenN; j += 256) {
      double z = j * R.dz;
      double a = u + R.c * z;
      double t0 = -1 / 2.0 * (a * a) - z;
      s = fma(exp(t0), green[(size_t)r * kSrGreenN + j], s);
    }
    s = warp_sum1(s);
    if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      double acc = 0.0;
      for (int w = 0; w < 8; ++w) acc += sw[w];
      total += R.coeff * (acc * R.dz);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) lag[(size_t)b * 3 * (2 * B - 1) + m + B - 1] = total;
  if (!green_t) return;
  // the transverse pseudo-Green wakes of the resonators (GetBBRPusdoWakeFun,
  // WakeFunction.cpp:596-629), for the potentials MPBunch.cpp:1981-1985
  // accumulates: per plane a header of CG_MAX_RESONATORS x (dz, 2Q/vz,
  // sqrt(2/pi) Rs c), then the resonators' sin(z a) / a tables
  for (int q = 0; q < 2; ++q) {
    const double* gt = green_t + (size_t)q * (3 * CG_MAX_RESONATORS + (size_t)n_res * kSrGreenN);
    double tq = 0.0;
    for (int r = 0; r < n_res; ++r) {
      const double dz = gt[3 * r], c = gt[3 * r + 1], coeff = gt[3 * r + 2];
      double s = 0.0;
      for (int j = threadIdx.x; j < kSrGreenN; j += 256) {
        double z = j * dz;
        double a = u + c * z;
        double t0 = -1 / 2.0 * (a * a) - z;
        s = fma(exp(t0), gt[3 * CG_MAX_RESONATORS + (size_t)r * kSrGreenN + j], s);
      }
      s = warp_sum1(s);
      if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = s;
      __syncthreads();
      if (threadIdx.x == 0) {
        double acc = 0.0;
        for (int w = 0; w < 8; ++w) acc += sw[w];
        tq += c * acc * dz * coeff;
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) lag[((size_t)b * 3 + 1 + q) * (2 * B - 1) + m + B - 1] = tq;
  }
}

// CTAs [0, n_chunks): a chunk each; then for each bunch CTAs of `per` lags.
template <bool XY>
__global__ void __launch_bounds__(kTile) k_sr_bins(const double* __restrict__ c, int64_t npad,
                                                   const uint8_t* __restrict__ surv,
                                                   const int4* __restrict__ chunk_loc, int n_chunks,
                                                   const BunchDev* __restrict__ bunch,
                                                   const BunchMomDev* __restrict__ mom, SrDev sr,
                                                   double* geom,
                                                   const SrResonator* __restrict__ res,
                                                   const double* __restrict__ green, int n_res,
                                                   double sigmat, double rw_coeff, double* lag,
                                                   const double* __restrict__ green_t, int per) {
  extern __shared__ unsigned char sm_raw[];
  const int B = sr.B, lags = 2 * B - 1, shares = (lags + per - 1) / per;
  const bool hist = (int)blockIdx.x < n_chunks;
  const int q = (int)blockIdx.x - n_chunks;
  const int4 l = hist ? chunk_loc[blockIdx.x] : make_int4(q / shares, 0, 0, 0);
  const int b = l.x, tile_off = bunch[b].tile_off;
  if (bunch[b].n_tiles == 0) return;  // held by another rank
  const SrGeom G = sr_geometry(sr.span[b], c[4 * npad + (int64_t)tile_off * kTile],
                               mom[b].bunch_length, B);
  if (hist) {
    sr_hist_chunk<XY>(c, npad, surv, l, bunch[b].n, tile_off, G, sr.counts + (size_t)b * B,
                      sr.sumx + (size_t)b * B, sr.sumy + (size_t)b * B, B, sm_raw);
    return;
  }
  const int m0 = q % shares * per;
  if (m0 == 0 && threadIdx.x == 0) {
    geom[2 * b] = G.lo;
    geom[2 * b + 1] = G.dz;
  }
  for (int m = m0; m < min(m0 + per, lags); ++m)
    sr_lag_cta(b, m - (B - 1), G.dz, res, green, n_res, B, sigmat, rw_coeff, lag, XY ? green_t : nullptr);
}

__global__ void __launch_bounds__(kTile) k_sr_pot(const BunchDev* __restrict__ bunch, SrDev sr,
                                                  const double* __restrict__ lag, double* pot,
                                                  double energy, double* potxy) {
  const int b = blockIdx.y, B = sr.B;
  if (bunch[b].n_tiles == 0) return;  // held by another rank
  const int i = blockIdx.x * (kTile / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (blockIdx.x == 0 && threadIdx.x == 0) sr.span[b] = SrSpan{0, 0};  // for the next call
  if (i >= B) return;
  const int* cnt = sr.counts + (size_t)b * B;
  const double* lg = lag + (size_t)b * 3 * (2 * B - 1) + i + B - 1;
  const double scale = (-1) * kElectronCharge * bunch[b].q_macro / energy;
  double v = 0, vx = 0, vy = 0;
  for (int j = lane; j < B; j += 32) {
    const int n = cnt[j];
    v += lg[-j] * n;
    if (!potxy) continue;
    // the transverse potentials, both from the horizontal centroids
    // (averXAlongBunch in both lines, MPBunch.cpp:1981-1985)
    const double ax = n ? sr.sumx[(size_t)b * B + j] / n : 0.0;
    vx += lg[(2 * B - 1) - j] * n * ax;
    vy += lg[2 * (2 * B - 1) - j] * n * ax;
  }
  v = warp_sum1(v);
  if (lane == 0) pot[(size_t)b * B + i] = (pot[(size_t)b * B + i] + v) * scale;
  if (!potxy) return;
  vx = warp_sum1(vx);
  vy = warp_sum1(vy);
  if (lane == 0) {
    double *px = potxy + (size_t)b * 2 * B + i, *py = px + B;
    *px = (*px + vx) * scale;
    *py = (*py + vy) * scale;
  }
}

template <bool MARK>
__global__ void __launch_bounds__(kTile) k_sr_kick(double* __restrict__ c, int64_t npad,
                                                   uint8_t* __restrict__ surv,
                                                   const int* __restrict__ tile_bunch,
                                                   const BunchDev* __restrict__ bunch,
                                                   const double* __restrict__ geom,
                                                   const double* __restrict__ pot, int B,
                                                   const __grid_constant__ Aperture ap,
                                                   int* loss_count) {
  const int b = tile_bunch[blockIdx.x];
  const BunchDev& Bd = bunch[b];
  const int64_t g = (int64_t)blockIdx.x * kTile + threadIdx.x;
  const bool valid = (blockIdx.x - Bd.tile_off) * kTile + (int)threadIdx.x < Bd.n;
  double x = 0, y = 0, z = 0;
  if (valid) {
    z = c[4 * npad + g];
    if (MARK) {
      x = c[g];
      y = c[2 * npad + g];
    }
    if (surv[g] == kAlive) {
      const double lo = geom[2 * b], dz = geom[2 * b + 1];
      const int idx = sr_bin(z, lo, dz, 1.0 / dz, B);
      if (idx >= 0) c[5 * npad + g] += pot[(size_t)b * B + idx];
    }
  }
  if (MARK) mark_lost_warp(ap, valid, x, y, z, surv + g, loss_count + b);
}

size_t sr_span_bytes() { return sizeof(SrSpan); }

SrDev sr_dev(const Handle& h) {
  return {reinterpret_cast<SrSpan*>(h.d.sr_span), h.d.sr_counts, h.d.sr_sumx, h.d.sr_sumy,
          h.cfg.sr_bins};
}

cudaError_t launch_sr_wake(Handle& h, bool have_range, bool mark) {
  const SrDev sr = sr_dev(h);
  const int B = sr.B;
  if (!have_range)
    k_sr_range<<<h.n_tiles, kTile, 0, h.stream>>>(h.d.c, h.npad, h.d.surv, h.d.tile_bunch,
                                                  h.d.bunch, sr);
  const double sigmat = 1.e-3 / kCLight;
  const bool xy = h.sr_xy && h.d.sr_potxy;
  const size_t sm = ((B * sizeof(int) + 15) & ~(size_t)15) + (xy ? 2 * B * sizeof(double) : 0);
  // lags per CTA: one while a few rounds of the 1184 CTAs that run at once hold
  // them all; beyond, a CTA's start (three loads, one after the other) would
  // cost as much as a lag (1000 bunches, 100 bins: a turn 2019 -> 1438 us)
  const int lags = 2 * B - 1;
  const int per = (int)std::min<int64_t>(lags, std::max<int64_t>(1, (int64_t)h.M * lags / (4 * 1184)));
  const int shares = (lags + per - 1) / per;
  (xy ? k_sr_bins<true> : k_sr_bins<false>)<<<h.n_chunks + h.M * shares, kTile, sm, h.stream>>>(
      h.d.c, h.npad, h.d.surv, h.d.chunk_loc, h.n_chunks, h.d.bunch, h.d.mom, sr, h.d.sr_geom,
      reinterpret_cast<const SrResonator*>(h.d.sr_green), h.d.sr_green + 3 * CG_MAX_RESONATORS,
      h.cfg.sr_bbr.n, sigmat, h.sr_rw_coeff, h.d.sr_lag, h.d.sr_green_t, per);
  k_sr_pot<<<dim3((B + kTile / 32 - 1) / (kTile / 32), h.M), kTile, 0, h.stream>>>(
      h.d.bunch, sr, h.d.sr_lag, h.d.sr_pot, h.cfg.ring.electron_energy, xy ? h.d.sr_potxy : nullptr);
  (mark ? k_sr_kick<true> : k_sr_kick<false>)<<<h.n_tiles, kTile, 0, h.stream>>>(
      h.d.c, h.npad, h.d.surv, h.d.tile_bunch, h.d.bunch, h.d.sr_geom, h.d.sr_pot, B, aperture(h),
      h.d.loss_count);
  return cudaGetLastError();
}

}  // namespace cg
