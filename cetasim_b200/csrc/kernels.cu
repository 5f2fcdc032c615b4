// sm_100a kernels of the MP tracking path.
//
// Data layout in HBM: six FP64 structure-of-arrays coordinate vectors
// (x, px, y, py, z, dp), each of `npad` doubles, plus one survival byte per
// particle.  Bunch j occupies tiles [tile_off[j], tile_off[j] + n_tiles[j]);
// every bunch segment starts on a 256-particle tile boundary (2 KiB), so
// loads of one CTA are fully coalesced 128-byte lines and a tile never spans
// two bunches.  Bunches of uneven size (ragged trains) are just different
// tile counts; fill-pattern gaps hold no tiles at all.
#include <cuda_runtime.h>
#include <algorithm>
#include "kernels.cuh"
#include "normals.cuh"
#include "turn_tail.cuh"

namespace cg {

#define FULL_MASK 0xffffffffu

// ---------------------------------------------------------------------------
// Block reductions with a fixed combination tree (deterministic results).

template <int N>
__device__ __forceinline__ void warp_sum(double (&v)[N]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] += __shfl_xor_sync(FULL_MASK, v[k], o);
}

// Sum N values over a CTA of NT threads; every thread receives the totals.
// smem must hold N * 32 doubles.
template <int N, int NT>
__device__ __forceinline__ void block_sum(double (&v)[N], double* smem) {
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  warp_sum<N>(v);
  if (NW == 1) return;
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < N; ++k) smem[k * 32 + warp] = v[k];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = (lane < NW) ? smem[k * 32 + lane] : 0.0;
    warp_sum<N>(v);
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < N; ++k) smem[k * 32] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = smem[k * 32];
  __syncthreads();
}

// Warp sums of 8 values with the transposed butterfly: at the shuffles by 16,
// 8 and 4 each lane passes half of its remaining values to its partner and
// keeps the other half, then the last value is summed by 2 and 1.  18
// shuffles of a double instead of 40; afterwards lane l holds the warp total
// of value ((l >> 4) & 1) * 4 + ((l >> 3) & 1) * 2 + ((l >> 2) & 1).  Fixed
// tree: deterministic.
__device__ __forceinline__ double warp_sum8_t(const double (&v)[8]) {
  const int lane = threadIdx.x & 31;
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
  double k4[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double keep = b4 ? v[i + 4] : v[i], send = b4 ? v[i] : v[i + 4];
    k4[i] = keep + __shfl_xor_sync(FULL_MASK, send, 16);
  }
  double k2[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double keep = b3 ? k4[i + 2] : k4[i], send = b3 ? k4[i] : k4[i + 2];
    k2[i] = keep + __shfl_xor_sync(FULL_MASK, send, 8);
  }
  const double keep = b2 ? k2[1] : k2[0], send = b2 ? k2[0] : k2[1];
  double t = keep + __shfl_xor_sync(FULL_MASK, send, 4);
  t += __shfl_xor_sync(FULL_MASK, t, 2);
  t += __shfl_xor_sync(FULL_MASK, t, 1);
  return t;
}
__device__ __forceinline__ int warp_sum8_index(int lane) {
  return ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
}

template <int NT>
__device__ __forceinline__ void block_minmax(double& mn, double& mx, double* smem) {
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = fmin(mn, __shfl_xor_sync(FULL_MASK, mn, o));
    mx = fmax(mx, __shfl_xor_sync(FULL_MASK, mx, o));
  }
  if (NW == 1) return;
  if (lane == 0) {
    smem[warp] = mn;
    smem[32 + warp] = mx;
  }
  __syncthreads();
  if (warp == 0) {
    mn = lane < NW ? smem[lane] : INFINITY;
    mx = lane < NW ? smem[32 + lane] : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn = fmin(mn, __shfl_xor_sync(FULL_MASK, mn, o));
      mx = fmax(mx, __shfl_xor_sync(FULL_MASK, mx, o));
    }
    if (lane == 0) {
      smem[0] = mn;
      smem[32] = mx;
    }
  }
  __syncthreads();
  mn = smem[0];
  mx = smem[32];
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Tile addressing

struct TileIdx {
  int b;       // bunch
  int i;       // index within the bunch
  int64_t g;   // global index into the SoA arrays
  bool valid;  // i < n_b
};

__device__ __forceinline__ TileIdx tile_index(const int* tile_bunch, const BunchDev* bunch) {
  TileIdx t;
  t.b = tile_bunch[blockIdx.x];
  const BunchDev& B = bunch[t.b];
  t.i = (blockIdx.x - B.tile_off) * kTile + threadIdx.x;
  t.g = (int64_t)blockIdx.x * kTile + threadIdx.x;
  t.valid = t.i < B.n;
  return t;
}

__device__ __forceinline__ void load6(const double* __restrict__ c, int64_t npad, int64_t g,
                                      double v[6]) {
#pragma unroll
  for (int d = 0; d < 6; ++d) v[d] = c[d * npad + g];
}
__device__ __forceinline__ void store6(double* __restrict__ c, int64_t npad, int64_t g,
                                       const double v[6]) {
#pragma unroll
  for (int d = 0; d < 6; ++d) c[d * npad + g] = v[d];
}

// ---------------------------------------------------------------------------
// Moments (MPBunch::GetMPBunchRMS, MPBunch.cpp:342-498): a CTA takes a chunk
// (consecutive tiles of one bunch) and each thread adds up its particles of
// the chunk as deviations from its warp's pivot, the mean of the first 32 that
// hold an alive particle, so that one pass over the particles is as accurate
// as the reference's two (the pivot lies within a fraction of sigma of the
// mean).  Each warp stores its sums as a partial (count, means, centred
// co-moments) and is done; k_mom_merge, one CTA per bunch, merges a bunch's
// partials in a fixed order: deterministic.  (A merge by the last CTA of each
// bunch costs every CTA a fence and an atomic: some 5 us at the end of each.)
// The map pass and k_moments share these functions: the same moments bit for
// bit.

template <class Count>
struct MomSumsOf {
  double s[6], q[9], zmin, zmax;
  Count n;
};
using MomSums = MomSumsOf<int>;
template <class Count>
__device__ __forceinline__ void mom_sums_clear(MomSumsOf<Count>& m) {
#pragma unroll
  for (int d = 0; d < 6; ++d) m.s[d] = 0.0;
#pragma unroll
  for (int k = 0; k < 9; ++k) m.q[k] = 0.0;
  m.zmin = INFINITY;
  m.zmax = -INFINITY;
  m.n = 0;
}
// ZR: the z range too
template <bool ZR>
__device__ __forceinline__ void mom_sums_add(MomSums& m, const double (&v)[6], const double* pivot) {
  double d[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    d[k] = v[k] - pivot[k];
    m.s[k] += d[k];
    m.q[k] = fma(d[k], d[k], m.q[k]);
  }
  m.q[6] = fma(d[0], d[1], m.q[6]);
  m.q[7] = fma(d[2], d[3], m.q[7]);
  m.q[8] = fma(d[4], d[5], m.q[8]);
  if (ZR) {
    m.zmin = fmin(m.zmin, v[4]);
    m.zmax = fmax(m.zmax, v[4]);
  }
  m.n += 1;
}

// Threads of a CTA of the map pass and the moments, and its steps per tile.
constexpr int kPassThreads = 128;
constexpr int kPassSteps = kTile / kPassThreads;
static_assert(kMomWarps * 32 == kPassThreads, "one partial per warp");

// Sets the warp's pivot if some lane's particle is alive; the warp calls it
// per tile until it returns true.  The pivot is the mean of the warp's alive
// particles, or the first one where that is the same to rounding: a coordinate
// that is equal in all of them has deviations of exactly zero.
__device__ __forceinline__ bool mom_pivot(double* pivot, bool alive, const double (&v)[6]) {
  const unsigned bal = __ballot_sync(FULL_MASK, alive);
  if (!bal) return false;
  const int lane = threadIdx.x & 31, idx = warp_sum8_index(lane);
  double a[8];
  if (lane == __ffs(bal) - 1)
#pragma unroll
    for (int d = 0; d < 6; ++d) pivot[d] = v[d];
#pragma unroll
  for (int d = 0; d < 6; ++d) a[d] = alive ? v[d] : 0.0;
  a[6] = a[7] = 0.0;
  const double t = warp_sum8_t(a);
  __syncwarp();
  if ((lane & 3) == 0 && idx < 6) {
    const double mean = t / __popc(bal);
    if (fabs(mean - pivot[idx]) > 1e-14 * fabs(mean)) pivot[idx] = mean;
  }
  __syncwarp();
  return true;
}

// The warp's sums as a partial.
template <class Count>
__device__ __forceinline__ void mom_partial(const MomSumsOf<Count>& m, bool have, const double* pivot,
                                            MomPartial* out) {
  const int lane = threadIdx.x & 31;
  // lane 4 i gets total i: s 0..5, n, q8, and q 0..7
  const double a[8] = {m.s[0], m.s[1], m.s[2], m.s[3], m.s[4], m.s[5], (double)m.n, m.q[8]};
  const double b[8] = {m.q[0], m.q[1], m.q[2], m.q[3], m.q[4], m.q[5], m.q[6], m.q[7]};
  const double t = warp_sum8_t(a), q = warp_sum8_t(b);
  double mn = m.zmin, mx = m.zmax;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = fmin(mn, __shfl_xor_sync(FULL_MASK, mn, o));
    mx = fmax(mx, __shfl_xor_sync(FULL_MASK, mx, o));
  }
  const double n = __shfl_sync(FULL_MASK, t, 24);
  const double inv = n > 0 ? 1.0 / n : 0.0;
  // co-moment k of lane 4 k: its pair of coordinates
  const int k = lane >> 2;
  const int i = k < 6 ? k : 2 * (k - 6), j = k < 6 ? k : 2 * (k - 6) + 1;
  const double si = __shfl_sync(FULL_MASK, t, 4 * i), sj = __shfl_sync(FULL_MASK, t, 4 * j);
  const double s4 = __shfl_sync(FULL_MASK, t, 16), s5 = __shfl_sync(FULL_MASK, t, 20);
  if ((lane & 3) == 0) {
    out->c[k] = q - si * (sj * inv);
    if (k < 6) out->mean[k] = have ? pivot[k] + t * inv : 0.0;
    else if (k == 6) out->n = n;
    else out->c[8] = t - s4 * (s5 * inv);
  }
  if (lane == 1) out->zmin = mn;
  if (lane == 2) out->zmax = mx;
}

// A warp merges every stride-th 32 of n_parts partials from `at` on in one pass:
// sums about the mean of the first non-empty one of its first round with any
// (means that are the same in all stay that value exactly; the co-moments'
// correction is as small as that mean is close).  GLOBAL: perhaps written by
// other CTAs of this launch, read through L2.
template <bool GLOBAL>
__device__ __forceinline__ void mom_merge_warp(const MomPartial* partials, int n_parts, int at,
                                               int stride, double* pivot, MomPartial* out) {
  auto get = [](const double* p) { return GLOBAL ? __ldcg(p) : *p; };
  const int lane = threadIdx.x & 31;
  MomSumsOf<double> m;
  mom_sums_clear(m);
  bool have = false;
  for (; at < n_parts; at += stride) {
    const MomPartial* p = partials + at + lane;
    const bool valid = at + lane < n_parts;
    const double n = valid ? get(&p->n) : 0.0;
    double d[6], c[9];
#pragma unroll
    for (int k = 0; k < 6; ++k) d[k] = valid ? get(&p->mean[k]) : 0.0;
#pragma unroll
    for (int k = 0; k < 9; ++k) c[k] = valid ? get(&p->c[k]) : 0.0;
    const double zmin = valid ? get(&p->zmin) : INFINITY, zmax = valid ? get(&p->zmax) : -INFINITY;
    if (!have) {
      const unsigned bal = __ballot_sync(FULL_MASK, n > 0);
      if (lane == __ffs(bal) - 1)
#pragma unroll
        for (int k = 0; k < 6; ++k) pivot[k] = d[k];
      __syncwarp();
      have = bal != 0;
    }
    m.zmin = fmin(m.zmin, zmin);
    m.zmax = fmax(m.zmax, zmax);
    if (!(n > 0)) continue;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      d[k] -= pivot[k];
      m.s[k] = fma(n, d[k], m.s[k]);
      m.q[k] += fma(n * d[k], d[k], c[k]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) m.q[6 + k] += fma(n * d[2 * k], d[2 * k + 1], c[6 + k]);
    m.n += n;
  }
  mom_partial(m, have, pivot, out);
}

// A CTA of NT threads merges n_parts partials: the warps their shares, then one
// warp the warps' results.  Every thread of the CTA calls it; warp 0 may read
// the result.
template <int NT, bool GLOBAL = true>
__device__ __forceinline__ const MomPartial* mom_merge_block(const MomPartial* partials, int n_parts) {
  constexpr int NW = NT / 32;
  __shared__ MomPartial s_part[NW + 1];
  __shared__ double s_pivot[NW][6];
  const int warp = NW > 1 ? (int)threadIdx.x >> 5 : 0;
  mom_merge_warp<GLOBAL>(partials, n_parts, warp * 32, NT, s_pivot[warp], &s_part[warp]);
  if (NW == 1) {
    __syncwarp();
    return s_part;
  }
  __syncthreads();
  if (warp == 0) {
    mom_merge_warp<false>(s_part, NW, 0, 32, s_pivot[0], &s_part[NW]);
    __syncwarp();
  }
  return s_part + NW;
}

// One CTA of NT threads per bunch: its partials merged and finalised.  z0 = z of
// the bunch's first particle (GetZMinMax seeds the range with it,
// MPBunch.cpp:1862-1863).
template <int NT>
__global__ void __launch_bounds__(NT) k_mom_merge(const double* __restrict__ c, int64_t npad,
                                                  const BunchDev* __restrict__ bunch,
                                                  const MomPartial* partials, BunchMomDev* mom,
                                                  double beta_x, double beta_y) {
  const int b = blockIdx.x;
  const BunchDev& B = bunch[b];
  if (B.n_chunks == 0) return;  // held by another rank
  const MomPartial* total =
      mom_merge_block<NT>(partials + (size_t)B.chunk_off * kMomWarps, B.n_chunks * kMomWarps);
  if (threadIdx.x != 0) return;
  BunchMomDev m;
  mom_finalize(*total, beta_x, beta_y, c[4 * npad + (int64_t)B.tile_off * kTile], m);
  m.transmission = mom[b].transmission;
  m.pad = 0.0;
  mom[b] = m;
}

// A warp per bunch while it has at most eight rounds of partials to read.
cudaError_t launch_mom_merge(Handle& h, int k, cudaStream_t s) {
  const SectionDev& sec = h.sec_dev_host[k];
  auto kern = h.max_chunks * kMomWarps <= 8 * 32 ? k_mom_merge<32> : k_mom_merge<256>;
  kern<<<h.M, h.max_chunks * kMomWarps <= 8 * 32 ? 32 : 256, 0, s ? s : h.stream>>>(
      h.d.c, h.npad, h.d.bunch, h.d.wpartials, h.d.mom, sec.beta_x, sec.beta_y);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(kPassThreads, 6) k_moments(const double* __restrict__ c,
                                                          int64_t npad,
                                                          const uint8_t* __restrict__ surv,
                                                          const int4* __restrict__ chunk_loc,
                                                          MomPartial* partials) {
  __shared__ double s_pivot[kMomWarps][6];
  const int4 l = chunk_loc[blockIdx.x];
  int64_t g = (int64_t)l.y * kTile + threadIdx.x;
  const int warp = threadIdx.x >> 5;
  MomSums m;
  mom_sums_clear(m);
  bool have = false;
#pragma unroll 1
  for (int u = 0; u < kPassSteps * l.z; ++u, g += kPassThreads) {
    const bool alive = surv[g] == kAlive;
    double w[6];
    load6(c, npad, g, w);
    if (!have) have = mom_pivot(s_pivot[warp], alive, w);
    if (alive) mom_sums_add<true>(m, w, s_pivot[warp]);
  }
  mom_partial(m, have, s_pivot[warp], &partials[(size_t)blockIdx.x * kMomWarps + warp]);
}

cudaError_t launch_moments(Handle& h, int k) {
  if (h.n_chunks < 1) return cudaSuccess;
  k_moments<<<h.n_chunks, kPassThreads, 0, h.stream>>>(h.d.c, h.npad, h.d.surv, h.d.chunk_loc,
                                                       h.d.wpartials);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = launch_mom_merge(h, k, h.stream);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Section map (Bunch::BunchTransferDueToLatticeTSymplectic) of the tiles from
// tile_base on, a thread per particle: the pass of a section whose moments
// nothing reads and where no ions kick.  Bound by HBM: every load of a particle
// at once (the padding slots hold the survival mark kPadding) and as many warps
// as the registers allow.  8.7e6 particles through a turn of 20 sections: 3.82 ms
// (5.00 as the moments' pass without the moments, 3.98 with four particles a
// thread in flight).

__global__ void __launch_bounds__(kTile) k_map(double* __restrict__ c, int64_t npad,
                                               const uint8_t* __restrict__ surv,
                                               const __grid_constant__ SectionDev sec,
                                               const __grid_constant__ RingDev r, int tile_base) {
  const int64_t g = (int64_t)(tile_base + (int)blockIdx.x) * kTile + threadIdx.x;
  const uint8_t alive = surv[g];
  double v[6];
  load6(c, npad, g, v);
  if (alive != kAlive) return;
  section_map_particle(sec, r, v);
  store6(c, npad, g, v);
}

cudaError_t launch_map(Handle& h, int k, int tile_a, int tile_b, cudaStream_t s) {
  if (tile_b < 0) tile_b = h.n_tiles;
  if (tile_b <= tile_a) return cudaSuccess;
  k_map<<<tile_b - tile_a, kTile, 0, s ? s : h.stream>>>(h.d.c, h.npad, h.d.surv, h.sec_dev_host[k],
                                                         h.ring, tile_a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Electron-side ion kick (MPBunch.cpp:1164-1206 + Bunch.cpp:213-220) with the
// cloud Gaussians the chain kernel recorded for each bunch at this IP.

// NT threads per CTA (a CTA covers NT particles of one tile) and at least
// MINB CTAs per SM (the register budget): the shapes the autotuner picks from.
template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_ion_kick(double* __restrict__ c, int64_t npad,
                                                      const uint8_t* __restrict__ surv,
                                                      const int* __restrict__ tile_bunch,
                                                      const CloudRec* __restrict__ rec,
                                                      const FieldPrep* __restrict__ rec_prep,
                                                      int P, int tile_base) {
  constexpr int kSub = kTile / NT;
  const int tile = tile_base + (int)(blockIdx.x / kSub);
  const int b = tile_bunch[tile];
  const int lane = (blockIdx.x % kSub) * NT + threadIdx.x;
  const int64_t g = (int64_t)tile * kTile + lane;  // padding slots hold kPadding
  __shared__ KickConst s_kc[CG_MAX_SPECIES];
  // every load of the particle at once (one memory round trip); the field
  // constants of the bunch's records come precomputed with the records
  rec += (size_t)b * P;
  rec_prep += (size_t)b * P;
  if ((int)threadIdx.x < P) s_kc[threadIdx.x] = kick_const(rec[threadIdx.x], rec_prep[threadIdx.x]);
  const uint8_t alive = surv[g];
  const double x = c[0 * npad + g], y = c[2 * npad + g];
  const double px = c[1 * npad + g], py = c[3 * npad + g];
  __syncthreads();
  if (alive != kAlive) return;
  double dpx, dpy;
  ion_kick_particle(s_kc, rec, rec_prep, P, x, y, &dpx, &dpy);
  c[1 * npad + g] = px + dpx;
  c[3 * npad + g] = py + dpy;
}

// The kick shapes of autotune choice v: threads per CTA and minimum CTAs per SM
// (the register budget).  Three kernels; the numbers 1 and 4 to 7 once stood
// for a 64-register shape, which spills, and for several tiles per CTA, which
// the occupancy of these makes needless (359 us against 361 for 1.74e7 kicks;
// 374 since two terms more of the series are in double precision).
static const int kKickShapes[][2] = {{256, 3}, {256, 3}, {128, 4}, {128, 6},
                                     {256, 3}, {128, 6}, {128, 6}, {256, 3}};
constexpr int kKickVariants = 8;

cudaError_t launch_ion_kick_variant(Handle& h, int k, int v, int tile_a, int tile_b,
                                    cudaStream_t s) {
  const CloudRec* rec = h.d.rec + (size_t)k * h.M * h.P;
  const FieldPrep* rp = h.d.rec_prep + (size_t)k * h.M * h.P;
  if (tile_b < 0) tile_b = h.n_tiles;
  if (!s) s = h.stream;
  const int nt = tile_b - tile_a;
  if (nt <= 0) return cudaSuccess;
  const int* shape = kKickShapes[v];
  switch (shape[0] == 128 ? shape[1] : 0) {
    case 4:
      k_ion_kick<128, 4><<<2 * nt, 128, 0, s>>>(h.d.c, h.npad, h.d.surv, h.d.tile_bunch,
                                                rec, rp, h.P, tile_a);
      break;
    case 6:
      k_ion_kick<128, 6><<<2 * nt, 128, 0, s>>>(h.d.c, h.npad, h.d.surv, h.d.tile_bunch,
                                                rec, rp, h.P, tile_a);
      break;
    default:
      k_ion_kick<256, 3><<<nt, 256, 0, s>>>(h.d.c, h.npad, h.d.surv, h.d.tile_bunch, rec, rp,
                                            h.P, tile_a);
  }
  return cudaGetLastError();
}

int kick_variants() { return kKickVariants; }
int kick_variant_first(int v) {
  int u = 0;
  while (kKickShapes[u][0] != kKickShapes[v][0] || kKickShapes[u][1] != kKickShapes[v][1]) ++u;
  return u;
}

// The particles' pass of one interaction point: the electron-side ion kick
// (KICK), the map of section k and the moments the next stage reads (MOM: at
// the twiss of section `mom_section`, MPBeam.cpp:1061/1069), each particle
// read and written once.  A CTA takes one chunk, half a tile after the other;
// other warps run while one's loads are under way.  Results equal k_ion_kick,
// k_map and k_moments in turn, bit for bit.
// Bound by issue: 805 instructions a particle of which 337 on the FP64 pipe (46 %
// busy) at 16 warps an SM, the accumulators of the moments beside the two
// series leaving no registers for more: 128 a thread spill 44 bytes (one
// instruction in fifty).  1.74e7 particles: 627 us (kick 374 and map with
// moments 404 apart; 471 and 441 before); floors 326 us of FP64 and 260 us of
// HBM.  Two particles at a time spill more (810 us); the next tile's loads in
// registers or by cp.async gain nothing (660 us); an unrolled loop misses the
// instruction cache (729 us).  Without the kick five CTAs per SM spill 140 bytes
// at 96 registers; four that spill nothing took 4013 us for a turn of the 32 x 32
// space charge instead of 3953.
// MOM: 0 no moments, 1 moments without the z range (which only the turn's last
// moments, the ones that callers can read, need), 2 all.
template <int MOM, bool KICK>
__global__ void __launch_bounds__(kPassThreads, KICK ? 4 : 5) k_map_pass(double* __restrict__ c,
                                                    int64_t npad, const uint8_t* __restrict__ surv,
                                                    const int4* __restrict__ chunk_loc,
                                                    const __grid_constant__ SectionDev sec,
                                                    const __grid_constant__ RingDev r,
                                                    MomPartial* partials,
                                                    const CloudRec* __restrict__ rec,
                                                    const FieldPrep* __restrict__ rec_prep, int P,
                                                    int chunk_base) {
  __shared__ double s_pivot[kMomWarps][6];
  __shared__ KickConst s_kc[KICK ? CG_MAX_SPECIES : 1];
  const int chunk = chunk_base + (int)blockIdx.x;
  // the chunk's place from one table load (x bunch, y first tile, z tiles), so
  // the coordinate loads wait for one round trip; the padding slots of a tile
  // hold the survival mark kPadding
  const int4 l = chunk_loc[chunk];
  int64_t g = (int64_t)l.y * kTile + threadIdx.x;
  rec += (size_t)l.x * P;
  rec_prep += (size_t)l.x * P;
  if (KICK) {
    if ((int)threadIdx.x < P) s_kc[threadIdx.x] = kick_const(rec[threadIdx.x], rec_prep[threadIdx.x]);
    __syncthreads();
  }
  const int warp = threadIdx.x >> 5;
  MomSums m;
  if (MOM) mom_sums_clear(m);
  bool have = false;
#pragma unroll 1
  for (int u = 0; u < kPassSteps * l.z; ++u, g += kPassThreads) {
    const bool alive = surv[g] == kAlive;
    double w[6];
    load6(c, npad, g, w);
    if (alive) {
      if (KICK) {
        double dpx, dpy;
        ion_kick_particle(s_kc, rec, rec_prep, P, w[0], w[2], &dpx, &dpy);
        w[1] += dpx;
        w[3] += dpy;
      }
      section_map_particle(sec, r, w);
      store6(c, npad, g, w);
    }
    if (MOM) {
      if (!have) have = mom_pivot(s_pivot[warp], alive, w);
      if (alive) mom_sums_add<MOM == 2>(m, w, s_pivot[warp]);
    }
  }
  if (MOM) mom_partial(m, have, s_pivot[warp], &partials[(size_t)chunk * kMomWarps + warp]);
}

cudaError_t launch_map_pass(Handle& h, int k, int mom_section, bool kick, bool z_range,
                            int chunk_a, int chunk_b, cudaStream_t s) {
  const int m = mom_section < 0 ? 0 : z_range ? 2 : 1;
  const CloudRec* rec = kick ? h.d.rec + (size_t)k * h.M * h.P : nullptr;
  const FieldPrep* rp = kick ? h.d.rec_prep + (size_t)k * h.M * h.P : nullptr;
  const bool all = chunk_b < 0;
  if (all) chunk_b = h.n_chunks;
  if (!s) s = h.stream;
  if (chunk_b > chunk_a) {
    if (!m && !kick) return cudaErrorInvalidValue;
    auto kern = m == 2   ? (kick ? k_map_pass<2, true> : k_map_pass<2, false>)
                : m == 1 ? (kick ? k_map_pass<1, true> : k_map_pass<1, false>)
                         : k_map_pass<0, true>;
    kern<<<chunk_b - chunk_a, kPassThreads, 0, s>>>(h.d.c, h.npad, h.d.surv, h.d.chunk_loc,
                                                    h.sec_dev_host[k], h.ring, h.d.wpartials, rec,
                                                    rp, h.P, chunk_a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return m && all ? launch_mom_merge(h, mom_section, s) : cudaSuccess;
}

cudaError_t launch_ion_kick(Handle& h, int k) { return launch_ion_kick_variant(h, k, h.kick_variant); }

// ---------------------------------------------------------------------------
// Turn tail: RF kick, drift, energy loss (all particles), synchrotron
// radiation (alive), long-range wake kick (all particles).

//
// Bound by instruction issue: the quantum excitation's three pairs of normals
// are half of the work.  With the library's log, square root and sincospi (and
// two divisions per cavity) a particle took 1016 instructions; the branch-free
// forms of normals.cuh take 725.  1.6e6 particles with one cavity:
// 73 -> 54 us.
//
// If nothing after it in the turn depends on the survival marks before the
// loss check (kLongMark), the check is made here on the final position; the
// bunches' counts end up in the transmission (k_turn_end).  If the broadband
// impedance (kLongBbi) or the short-range wake (kLongSr) comes next, the
// bunches' ranges that it starts from are collected.

//
// The ring's last map joins it where nothing reads the beam between the two (no
// moments, no kick, no beam loading): the particles are read and written once
// for both.  1.6e6 particles, with the broadband impedance's ranges: map
// 35 + 58 -> 69 us, the turn 149 -> 127 us.

// LOADING: some cavity has beam loading; TAIL: kLongMark, kLongBbi or kLongSr;
// MAP: the map of section `last` first
template <bool LOADING, unsigned TAIL, bool MAP = false>
__global__ void __launch_bounds__(kTile, 4) k_long(double* __restrict__ c, int64_t npad,
                                                  uint8_t* __restrict__ surv,
                                                  const int* __restrict__ tile_bunch,
                                                  const BunchDev* __restrict__ bunch,
                                                  const __grid_constant__ SectionDev sec0,
                                                  const __grid_constant__ RingDev r,
                                                  unsigned flags, uint64_t seed,
                                                  const int* __restrict__ d_turn,
                                                  const double* __restrict__ lr_force,
                                                  const double* __restrict__ rf_zr,
                                                  const double* __restrict__ rf_kick,
                                                  const double* __restrict__ rf_fbk, int M,
                                                  double* rf_info,
                                                  const __grid_constant__ Aperture ap,
                                                  int* loss_count,
                                                  const __grid_constant__ BbiParams bbi,
                                                  BbiSpan* span, int* status, const SrDev sr,
                                                  const __grid_constant__ SectionDev last) {
  TileIdx t = tile_index(tile_bunch, bunch);
  double v[6] = {0, 0, 0, 0, 0, 0};
  bool alive = false;
  if (t.valid) {
    load6(c, npad, t.g, v);
    alive = (LOADING || MAP || TAIL == kLongBbi || TAIL == kLongSr || (flags & kLongSynrad)) &&
            surv[t.g] == kAlive;
    if (MAP && alive) section_map_particle(last, r, v);
    if (flags & kLongRF) {
      if (t.i == bunch[t.b].n - 1) {
        // the ideal cavities' BunchRFModeInfo: the voltage the bunch's last
        // particle sees (Bunch.cpp:466-478; cavity = generator, no induced or
        // self-loss voltage)
        for (int q = 0; q < r.n_cav; ++q) {
          if (LOADING && r.bl_index[q] >= 0) continue;
          double sn, co;
          sincos_far(v[4] * r.rf_theta_coeff[q], &sn, &co);
          const double re = fma(r.vreq_re[q], co, r.vreq_im[q] * sn);
          const double im = fma(r.vreq_im[q], co, -r.vreq_re[q] * sn);
          double* o = rf_info + ((size_t)t.b * CG_MAX_CAVITIES + q) * 8;
          o[0] = re; o[1] = im; o[2] = re; o[3] = im;
          o[4] = 0.0; o[5] = 0.0; o[6] = 0.0; o[7] = 0.0;
        }
      }
      if (LOADING) v[5] = rf_kick_dp_loading(r, v[4], v[5], alive, t.b, M, rf_zr, rf_kick, rf_fbk);
      else v[5] = rf_kick_dp(r, v[4], v[5]);
    }
    if (flags & kLongDrift) v[4] = drift_z(r, v[4], v[5]);
    if (flags & kLongLoss) v[5] -= r.u0_term;
    if ((flags & kLongSynrad) && alive) {
      double g[6] = {0, 0, 0, 0, 0, 0};
      const bool excite = bunch[t.b].n != 1;
      if (excite && (r.qe_coeff[0] != 0 || r.qe_coeff[1] != 0 || r.qe_coeff[2] != 0))
        synrad_normals(seed, (uint32_t)t.i, (uint32_t)t.b, (uint32_t)(*d_turn), g);
      synrad_particle(sec0, r, v, g, excite);
    }
    if (flags & kLongLR) {
      const double* f = lr_force + 3 * t.b;
      v[1] += f[0];
      v[3] += f[1];
      v[5] += f[2];
    }
    store6(c, npad, t.g, v);
  }
  if (TAIL == kLongMark)
    mark_lost_warp(ap, t.valid, v[0], v[2], v[4], surv + t.g, loss_count + t.b);
  if (TAIL == kLongBbi)
    bbi_span_cta(bbi, span + t.b, status, t.valid && bunch[t.b].q_macro != 0, alive, v[0], v[2],
                 v[4]);
  if (TAIL == kLongSr) sr_span_cta(sr, t.b, (int)blockIdx.x == bunch[t.b].tile_off, alive, v[4]);
}

// The accumulated phase advance of the tracked bunches' particles
// (Bunch.cpp:715-731), before the map of the ring's last section: per
// particle the angles of the rotated normal-form vector, their decrease since
// the last turn (plus 2 pi when negative) added up.  ph[slot] holds per
// particle (previous x, y, z angles, accumulated x, y, z), 6 x n.
__global__ void __launch_bounds__(kTile) k_phase_adv(const double* __restrict__ c, int64_t npad,
                                                     const uint8_t* __restrict__ surv,
                                                     const int* __restrict__ tile_bunch,
                                                     const BunchDev* __restrict__ bunch,
                                                     const __grid_constant__ SectionDev sec,
                                                     const __grid_constant__ RingDev r,
                                                     const int* __restrict__ slot_of,
                                                     double* const* __restrict__ ph, int tile0) {
  const int tile = tile0 + blockIdx.x;
  const int b = tile_bunch[tile];
  const BunchDev& B = bunch[b];
  const int i = (tile - B.tile_off) * kTile + threadIdx.x;
  const int64_t g = (int64_t)tile * kTile + threadIdx.x;
  const int slot = slot_of[b];
  if (i >= B.n || slot < 0 || surv[g] != kAlive) return;  // the map skips lost particles
  double v[6], v2[6];
  load6(c, npad, g, v);
  section_map_rotated(sec, r, v, v2);
  double* P = ph[slot];
  const int n = B.n;
  for (int q = 0; q < 3; ++q) {
    const double cur = atan2(v2[2 * q + 1], v2[2 * q]);
    const double tmp = P[(size_t)q * n + i] - cur;
    P[(size_t)(3 + q) * n + i] += tmp >= 0 ? tmp : tmp + 2 * kPi;
    P[(size_t)q * n + i] = cur;
  }
}

// Bunch::InitialAccumPhaseAdV (Bunch.cpp:504-553): the angles of B1H1 . v at
// section 0, accumulated phases zero.
__global__ void __launch_bounds__(kTile) k_phase_init(const double* __restrict__ c, int64_t npad,
                                                      const int* __restrict__ tile_bunch,
                                                      const BunchDev* __restrict__ bunch,
                                                      const __grid_constant__ SectionDev sec0,
                                                      const int* __restrict__ slot_of,
                                                      double* const* __restrict__ ph) {
  TileIdx t = tile_index(tile_bunch, bunch);
  if (!t.valid) return;
  const int slot = slot_of[t.b];
  if (slot < 0) return;
  double v[6], v1[6];
  load6(c, npad, t.g, v);
  matvec6(sec0.b1h1, v, v1);
  double* P = ph[slot];
  const int n = bunch[t.b].n;
  for (int q = 0; q < 3; ++q) {
    P[(size_t)q * n + t.i] = atan2(v1[2 * q + 1], v1[2 * q]);
    P[(size_t)(3 + q) * n + t.i] = 0.0;
  }
}

cudaError_t launch_phase_init(Handle& h) {
  k_phase_init<<<h.n_tiles, kTile, 0, h.stream>>>(h.d.c, h.npad, h.d.tile_bunch, h.d.bunch,
                                                  h.sec_dev_host[0], h.d.phase_slot, h.d.phase_ptr);
  return cudaGetLastError();
}

cudaError_t launch_phase_adv(Handle& h, int ja, int jb, cudaStream_t s) {
  bool any = false;
  for (int j : h.phase_bunches) any = any || (j >= ja && j < jb);
  if (!any) return cudaSuccess;
  const int ta = h.tile_off[ja], tb = jb < h.M ? h.tile_off[jb] : h.n_tiles;
  k_phase_adv<<<tb - ta, kTile, 0, s ? s : h.stream>>>(
      h.d.c, h.npad, h.d.surv, h.d.tile_bunch, h.d.bunch, h.sec_dev_host[h.K - 1], h.ring,
      h.d.phase_slot, h.d.phase_ptr, ta);
  return cudaGetLastError();
}

Aperture aperture(const Handle& h) {
  const cg_section& s = h.sections[0];
  return {s.aperture_x, s.aperture_y, 1.0 / s.aperture_x, 1.0 / s.aperture_y, h.ring.z_loss};
}

cudaError_t launch_long(Handle& h, unsigned flags, bool map) {
  if ((flags & kLongRF) && h.ring.bl_any) {
    // the cavities' recurrence over the train first: the kicks of each bin
    cudaError_t e = launch_rf_beam_loading(h);
    if (e != cudaSuccess) return e;
  }
  auto pick = [&](auto none, auto mark, auto bbi, auto sr) {
    return flags & kLongMark ? mark : flags & kLongBbi ? bbi : flags & kLongSr ? sr : none;
  };
  auto kern = h.ring.bl_any ? pick(k_long<true, 0>, k_long<true, kLongMark>, k_long<true, kLongBbi>,
                                   k_long<true, kLongSr>)
                            : pick(k_long<false, 0>, k_long<false, kLongMark>,
                                   k_long<false, kLongBbi>, k_long<false, kLongSr>);
  // the short-range wake reads moments after the map, beam loading the beam
  if (map && (h.ring.bl_any || (flags & kLongSr))) return cudaErrorInvalidValue;
  if (map) kern = pick(k_long<false, 0, true>, k_long<false, kLongMark, true>,
                       k_long<false, kLongBbi, true>, k_long<false, 0, true>);
  kern<<<h.n_tiles, kTile, 0, h.stream>>>(h.d.c, h.npad, h.d.surv, h.d.tile_bunch, h.d.bunch,
                                          h.sec_dev_host[0], h.ring, flags, h.cfg.seed, h.d.turn,
                                          h.d.lr_force, h.d.rf_zr, h.d.rf_kick, h.d.rf_fbk, h.M,
                                          h.d.rf_info, aperture(h), h.d.loss_count, h.bbi,
                                          reinterpret_cast<BbiSpan*>(h.d.bbi_span), h.d.status,
                                          sr_dev(h), h.sec_dev_host[h.K - 1]);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Long-range wake (MPBeam::LRWakeBeamIntaction, MPBeam.cpp:3232-3349).
// k_lr_push stores this turn's centroids in the history ring; k_lr_force
// sums the tabulated wake over (turn n, source bunch i) for each bunch j.

__global__ void k_lr_push(const BunchMomDev* __restrict__ mom, double* hist, int* head, int T,
                          int M) {
  __shared__ int h;
  if (threadIdx.x == 0) {
    h = (*head + 1) % T;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < M; i += blockDim.x) {
    double* slot = hist + (size_t)h * 3 * M;
    slot[i] = mom[i].mean[0];
    slot[M + i] = mom[i].mean[2];
    slot[2 * M + i] = mom[i].mean[4];
  }
  __syncthreads();
  if (threadIdx.x == 0) *head = h;
}

__global__ void k_lr_force(const BunchMomDev* __restrict__ mom, const BunchDev* __restrict__ bunch,
                           const double* __restrict__ hist, const int* __restrict__ head,
                           const double* __restrict__ tab, int np, double dt, double tRF,
                           double scale, int T, int M, int H, double inv_c_beta,
                           double* lr_force, int* status) {
  __shared__ double smem[3 * 32];
  const int j = blockIdx.x;
  const int hd = *head;
  const int hj = bunch[j].harm;
  const double zj = mom[j].mean[4];
  double f[3] = {0.0, 0.0, 0.0};
  // enumerate (n, i) pairs of the reference's loop: n = 0 -> i < j;
  // n = T-1 -> i >= j; otherwise all i.
  const int64_t total = (int64_t)T * M;
  for (int64_t q = threadIdx.x; q < total; q += blockDim.x) {
    int n = (int)(q / M), i = (int)(q % M);
    if (n == 0 && i >= j) continue;
    if (n == T - 1 && i < j) continue;
    const double* hs = hist + (size_t)((hd - n + T) % T) * 3 * M;
    int nT = bunch[i].harm - hj - n * H;
    double tau = nT * tRF + (zj - hs[2 * M + i]) * inv_c_beta;
    double a = -tau / dt;
    // compared before the conversion, which saturates (or gives the smallest
    // integer for a NaN)
    if (tau > 0 || !(a >= 0 && a < np - 1)) {
      atomicOr(status, kStatusLrRange);
      continue;
    }
    const int idx = (int)a;
    double v1 = a - idx, v0 = 1 - v1;
    double ne = bunch[i].ne;
    double w0 = tab[idx] * v0 + tab[idx + 1] * v1;
    double w1 = tab[np + idx] * v0 + tab[np + idx + 1] * v1;
    double w2 = tab[2 * np + idx] * v0 + tab[2 * np + idx + 1] * v1;
    f[0] -= w0 * ne * hs[i];
    f[1] -= w1 * ne * hs[M + i];
    f[2] -= w2 * ne;
  }
  block_sum<3, 256>(f, smem);
  if (threadIdx.x == 0) {
    lr_force[3 * j + 0] = f[0] * scale;
    lr_force[3 * j + 1] = f[1] * scale;
    lr_force[3 * j + 2] = f[2] * scale;
  }
}

cudaError_t launch_lr_compute(Handle& h) {
  const cg_ring& r = h.cfg.ring;
  int T = h.cfg.lr_turns;
  k_lr_push<<<1, 256, 0, h.stream>>>(h.d.mom, h.d.lr_hist, h.d.lr_head, T, h.M);
  double tRF = r.t0 / (double)r.harmonics;
  double scale = kElectronCharge / r.electron_energy / (r.r_beta * r.r_beta);
  double inv_c_beta = 1.0 / kCLight / r.r_beta;
  k_lr_force<<<h.M, 256, 0, h.stream>>>(h.d.mom, h.d.bunch, h.d.lr_hist, h.d.lr_head, h.d.lr_tab,
                                        h.lr_np, h.lr_dt, tRF, scale, T, h.M, r.harmonics,
                                        inv_c_beta, h.d.lr_force, h.d.status);
  return cudaGetLastError();
}

cudaError_t launch_lr_kick(Handle& h) { return launch_long(h, kLongLR); }

// ---------------------------------------------------------------------------
// FIR bunch-by-bunch feedback (MPBeam::FIRBunchByBunchFeedback,
// MPBeam.cpp:2978-3090): history push + kick per bunch.

__global__ void k_fir_compute(const BunchMomDev* __restrict__ mom, double* hist, int* head,
                              const double* __restrict__ coeff, int order, int M, int mode,
                              double gain, double kx, double ky, double kf, double limit,
                              const int* __restrict__ d_turn, int n_sec, int4 se0, int4 se1,
                              int4 se2, int4 se3, double* kick) {
  const int turn = *d_turn;
  int starts[8] = {se0.x, se0.z, se1.x, se1.z, se2.x, se2.z, se3.x, se3.z};
  int ends[8] = {se0.y, se0.w, se1.y, se1.w, se2.y, se2.w, se3.y, se3.w};
  bool on = false;
  for (int q = 0; q < n_sec && q < 8; ++q)
    if (turn > starts[q] && turn < ends[q]) on = true;
  if (mode == 0) {
    for (int j = threadIdx.x; j < M; j += blockDim.x) {
      kick[3 * j + 0] = on ? -mom[j].mean[1] : 0.0;
      kick[3 * j + 1] = on ? -mom[j].mean[3] : 0.0;
      kick[3 * j + 2] = on ? -mom[j].mean[5] : 0.0;
    }
    return;
  }
  __shared__ int hd;
  if (threadIdx.x == 0) hd = (*head + 1) % order;
  __syncthreads();
  for (int j = threadIdx.x; j < M; j += blockDim.x) {
    double* slot = hist + (size_t)hd * 3 * M;
    slot[j] = mom[j].mean[0];
    slot[M + j] = mom[j].mean[2];
    slot[2 * M + j] = mom[j].mean[4];
  }
  __syncthreads();
  if (threadIdx.x == 0) *head = hd;
  for (int j = threadIdx.x; j < M; j += blockDim.x) {
    double a = 0, b = 0, cz = 0;
    if (on) {
      // q = 0 is the oldest sample (reference posxData[0])
      for (int q = 0; q < order; ++q) {
        const double* hs = hist + (size_t)((hd + 1 + q) % order) * 3 * M;
        a += coeff[order - q - 1] * hs[j];
        b += coeff[order + order - q - 1] * hs[M + j];
        cz += coeff[2 * order + order - q - 1] * hs[2 * M + j];
      }
      a = a * gain * kx;
      b = b * gain * ky;
      cz = cz * gain * kf;
      if (a > limit) a = limit;
      if (b > limit) b = limit;
      if (cz > limit) cz = limit;
    }
    kick[3 * j + 0] = a;
    kick[3 * j + 1] = b;
    kick[3 * j + 2] = cz;  // divided by beta^2 when applied
  }
}

cudaError_t launch_fir_compute(Handle& h) {
  const cg_fir_params& f = h.cfg.fir;
  int st[8] = {0}, en[8] = {0};
  for (int q = 0; q < f.n_sections && q < 8; ++q) {
    st[q] = f.start[q];
    en[q] = f.end[q];
  }
  int4 a = {st[0], en[0], st[1], en[1]}, b = {st[2], en[2], st[3], en[3]};
  int4 c = {st[4], en[4], st[5], en[5]}, d = {st[6], en[6], st[7], en[7]};
  k_fir_compute<<<1, 256, 0, h.stream>>>(h.d.mom, h.d.fir_hist, h.d.fir_head, h.d.fir_coeff,
                                         h.fir_order, h.M, f.mode, f.gain, f.kick_strength[0],
                                         f.kick_strength[1], f.kick_strength[2], h.fir_limit,
                                         h.d.turn, f.n_sections, a, b, c, d, h.d.fir_kick);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// FIR kick (all particles) + Bunch::MarkLostParticle (Bunch.cpp:172-200): a
// pass over x, y, z, bound by HBM latency (1.6e6 particles 23 -> 16 us; it used
// to sum each tile over the CTA, fence, and divide twice per particle).

__global__ void __launch_bounds__(kTile) k_mark_lost(double* __restrict__ c, int64_t npad,
                                                     uint8_t* __restrict__ surv,
                                                     const int* __restrict__ tile_bunch,
                                                     const BunchDev* __restrict__ bunch,
                                                     const __grid_constant__ Aperture ap, int mode,
                                                     const double* __restrict__ fir_kick,
                                                     double inv_beta2, int* loss_count, bool mark) {
  TileIdx t = tile_index(tile_bunch, bunch);
  if (t.valid && mode > 0) {
    const double* k = fir_kick + 3 * t.b;
    c[1 * npad + t.g] += k[0];
    c[3 * npad + t.g] += k[1];
    if (mode == 1) c[5 * npad + t.g] += k[2] * inv_beta2;
    else c[5 * npad + t.g] += k[2];
  }
  if (!mark) return;
  double x = 0, y = 0, z = 0;
  if (t.valid) {
    x = c[t.g];
    y = c[2 * npad + t.g];
    z = c[4 * npad + t.g];
  }
  mark_lost_warp(ap, t.valid, x, y, z, surv + t.g, loss_count + t.b);
}

cudaError_t launch_mark_lost(Handle& h, bool fir_kick, bool mark) {
  int mode = 0;
  if (fir_kick) mode = (h.cfg.fir.mode == 0) ? 2 : 1;
  double inv_beta2 = 1.0 / (h.cfg.ring.r_beta * h.cfg.ring.r_beta);
  k_mark_lost<<<h.n_tiles, kTile, 0, h.stream>>>(h.d.c, h.npad, h.d.surv, h.d.tile_bunch,
                                                 h.d.bunch, aperture(h), mode,
                                                 h.d.fir_kick, inv_beta2, h.d.loss_count, mark);
  return cudaGetLastError();
}

// After the loss check: the bunches' transmission, and the turn's end.
__global__ void k_turn_end(const BunchDev* __restrict__ bunch, int M, int* loss_count,
                           BunchMomDev* mom, int* status, int* turn, int advance) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b == 0) *turn += advance;
  if (b >= M || bunch[b].n_tiles == 0) return;  // no particles here: another rank's
  const int n = bunch[b].n;
  const double tr = (n - loss_count[b]) / (double)n;
  loss_count[b] = 0;
  mom[b].transmission = tr;
  if (tr < 0.5) atomicOr(status, kStatusTransmission);
}

cudaError_t launch_turn_end(Handle& h, bool advance) {
  k_turn_end<<<(h.M + 127) / 128, 128, 0, h.stream>>>(h.d.bunch, h.M, h.d.loss_count, h.d.mom,
                                                      h.d.status, h.d.turn, advance ? 1 : 0);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Seeded initial distribution: MPBunch::DistriGenerator type 3
// (MPBunch.cpp:134-277) with counter-based draws: (z, dp) Gaussian cut at
// 3 sigma jointly (MPBunch.cpp:134-152), transverse Gaussian cut at 3 sigma
// in (x/rX)^2 + (y/rY)^2 (MPBunch.cpp:254-260), plus dispersion
// (MPBunch.cpp:268-277).  The reference draws the 4-D action radially
// (GSSlover) and splits it uniformly between the planes; for a Gaussian beam
// that is the law of independent normals per plane, which is what is drawn
// here.  As in the reference a rejected draw is drawn again until one is
// accepted: each cut keeps 98.9 % of draws, so kGaussAttempts attempts all
// fail with probability below 1e-1900; if that ever happens the particle
// keeps the zero vector and the status word reports it (no draw outside the
// cut is ever kept).
constexpr uint32_t kGaussAttempts = 1024;

__global__ void __launch_bounds__(kTile) k_gaussian(double* __restrict__ c, int64_t npad,
                                                    uint8_t* __restrict__ surv,
                                                    const int* __restrict__ tile_bunch,
                                                    const BunchDev* __restrict__ bunch,
                                                    const SectionDev* __restrict__ sec0,
                                                    double emit_x, double emit_y, double sz,
                                                    double sdp, double r_beta2, uint64_t seed,
                                                    int* __restrict__ status) {
  TileIdx t = tile_index(tile_bunch, bunch);
  if (!t.valid) {
    surv[t.g] = kPadding;  // padding slot: never alive
#pragma unroll
    for (int d = 0; d < 6; ++d) c[d * npad + t.g] = 0.0;
    return;
  }
  const SectionDev& s = *sec0;
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32) ^ kStreamInitDist;
  bool ok_l = false, ok_t = false;
  double z = 0, dp = 0;
  for (uint32_t a = 0; a < kGaussAttempts && !ok_l; ++a) {
    u32x4 ctr = {{(uint32_t)t.i, (uint32_t)t.b, a, 0u}};
    double g0, g1;
    normal2(philox4x32_10(ctr, k0, k1), &g0, &g1);
    if (g0 * g0 + g1 * g1 < 9.0) {
      z = sz * g0;
      dp = sdp * g1 / r_beta2;
      ok_l = true;
    }
  }
  double rx = sqrt(emit_x * s.beta_x), ry = sqrt(emit_y * s.beta_y);
  double x = 0, px = 0, y = 0, py = 0;
  for (uint32_t a = 0; a < kGaussAttempts && !ok_t; ++a) {
    u32x4 ctr = {{(uint32_t)t.i, (uint32_t)t.b, a, 1u}};
    double g0, g1, g2, g3;
    normal2(philox4x32_10(ctr, k0, k1), &g0, &g1);
    ctr.v[3] = 2u;
    normal2(philox4x32_10(ctr, k0, k1), &g2, &g3);
    // normalised phase space (u, u') ~ N(0, emit) per plane
    const double ux = sqrt(emit_x) * g0, upx = sqrt(emit_x) * g1;
    const double uy = sqrt(emit_y) * g2, upy = sqrt(emit_y) * g3;
    const double tx = sqrt(s.beta_x) * ux, ty = sqrt(s.beta_y) * uy;
    if ((tx / rx) * (tx / rx) + (ty / ry) * (ty / ry) <= 9.0) {
      x = tx;
      px = (upx - s.alpha_x * ux) / sqrt(s.beta_x);
      y = ty;
      py = (upy - s.alpha_y * uy) / sqrt(s.beta_y);
      ok_t = true;
    }
  }
  if (!(ok_l && ok_t)) atomicOr(status, kStatusGaussCut);
  x += s.eta_x * dp;
  y += s.eta_y * dp;
  px += s.etap_x * dp;
  py += s.etap_y * dp;
  double v[6] = {x, px, y, py, z, dp};
  store6(c, npad, t.g, v);
  surv[t.g] = kAlive;
}

cudaError_t launch_gaussian(Handle& h, double emit_x, double emit_y, double sigma_z,
                            double sigma_dp, uint64_t seed) {
  double rb2 = h.cfg.ring.r_beta * h.cfg.ring.r_beta;
  k_gaussian<<<h.n_tiles, kTile, 0, h.stream>>>(h.d.c, h.npad, h.d.surv, h.d.tile_bunch,
                                                h.d.bunch, h.sec_dev, emit_x, emit_y, sigma_z,
                                                sigma_dp, rb2, seed, h.d.status);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// The ten second moments of MPBunch::GetEigenEmit (MPBunch.cpp:500-560) for
// one bunch: every particle (lost ones too), x, x', y, y' less the dispersion
// of section 0 times dp, products taken about zero (the reference sums its
// "means" with an int accumulator, MPBunch.cpp:516-519, so they stay zero),
// not yet divided by n.  One CTA: per-thread sums in particle order, then a
// fixed tree over the threads (deterministic).
__global__ void __launch_bounds__(kTile) k_eigen_sums(const double* __restrict__ c, int64_t npad,
                                                      const BunchDev* __restrict__ bunch, int j,
                                                      const SectionDev* __restrict__ sec0,
                                                      double* __restrict__ out) {
  __shared__ double sh[10][kTile];
  const BunchDev b = bunch[j];
  const SectionDev& s = *sec0;
  double a[10];
#pragma unroll
  for (int q = 0; q < 10; ++q) a[q] = 0.0;
  const int64_t base = (int64_t)b.tile_off * kTile;
  for (int i = threadIdx.x; i < b.n; i += kTile) {
    const int64_t g = base + i;
    const double dp = c[5 * npad + g];
    const double x = c[g] - s.eta_x * dp, xp = c[npad + g] - s.etap_x * dp;
    const double y = c[2 * npad + g] - s.eta_y * dp, yp = c[3 * npad + g] - s.etap_y * dp;
    a[0] += x * x;   a[1] += x * xp;  a[2] += x * y;   a[3] += x * yp;  a[4] += xp * xp;
    a[5] += xp * y;  a[6] += xp * yp; a[7] += y * y;   a[8] += y * yp;  a[9] += yp * yp;
  }
#pragma unroll
  for (int q = 0; q < 10; ++q) sh[q][threadIdx.x] = a[q];
  __syncthreads();
  for (int w = kTile / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w)
#pragma unroll
      for (int q = 0; q < 10; ++q) sh[q][threadIdx.x] += sh[q][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < 10) out[threadIdx.x] = sh[threadIdx.x][0];
}

cudaError_t launch_eigen_sums(Handle& h, int j, double* out) {
  k_eigen_sums<<<1, kTile, 0, h.stream>>>(h.d.c, h.npad, h.d.bunch, j, h.sec_dev, out);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Stateless evaluators.

__global__ void k_faddeeva(const double* __restrict__ zr, const double* __restrict__ zi,
                           double* wr, double* wi, int64_t n, bool general) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  cplx w = general ? w_general(zr[i], zi[i]) : w_quadrant1(zr[i], zi[i]);
  wr[i] = w.re;
  wi[i] = w.im;
}

cudaError_t launch_faddeeva(const double* zr, const double* zi, double* wr, double* wi, int64_t n,
                            bool general, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  k_faddeeva<<<(unsigned)blocks, 256, 0, s>>>(zr, zi, wr, wi, n, general);
  return cudaGetLastError();
}

__global__ void k_field(const double* __restrict__ x, const double* __restrict__ y,
                        const double* __restrict__ sx, const double* __restrict__ sy, double* fx,
                        double* fy, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  gaussian_field(x[i], y[i], sx[i], sy[i], &fx[i], &fy[i]);
}

cudaError_t launch_field(const double* x, const double* y, const double* sx, const double* sy,
                         double* fx, double* fy, int64_t n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  k_field<<<(unsigned)blocks, 256, 0, s>>>(x, y, sx, sy, fx, fy, n);
  return cudaGetLastError();
}

// FP64 FMA throughput probe: 8 independent register FMA chains per thread.
__global__ void __launch_bounds__(256) k_fp64_peak(double* out, int iters, double a, double b) {
  double r[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) r[q] = threadIdx.x * 1e-3 + q;
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int q = 0; q < 8; ++q) r[q] = fma(r[q], a, b);
  }
  double s = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) s += r[q];
  if (s == 123.456) out[0] = s;  // keeps the chains live
}

cudaError_t measure_fp64_peak(double* flops) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  double* out = nullptr;
  cudaError_t e = cudaMalloc(&out, sizeof(double));
  if (e != cudaSuccess) return e;
  const int blocks = sms * 8, threads = 256, iters = 4096;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  k_fp64_peak<<<blocks, threads>>>(out, 64, 0.999999, 1e-7);  // warm-up
  cudaEventRecord(e0);
  k_fp64_peak<<<blocks, threads>>>(out, iters, 0.999999, 1e-7);
  cudaEventRecord(e1);
  e = cudaEventSynchronize(e1);
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  if (e != cudaSuccess) return e;
  *flops = 2.0 * 8.0 * iters * (double)blocks * threads / (ms * 1e-3);
  return cudaGetLastError();
}

cudaError_t upload_weideman_table() {
  cudaError_t e = cudaMemcpyToSymbol(c_weideman, &h_weideman, sizeof(WeidemanTable));
  if (e == cudaSuccess) e = upload_weideman_table_ion();
  if (e == cudaSuccess) e = upload_weideman_table_sc();
  return e != cudaSuccess ? e : upload_weideman_table_sur();
}

// ---------------------------------------------------------------------------
// Moments of one bunch in the caller's device buffers without any device
// allocation.  A caller that owns the particle arrays and calls once per turn
// (another code's tracking loop, a PyTorch program whose caching allocator owns
// the device memory) cannot afford a cudaMalloc/cudaFree pair per call: both
// synchronise the device and stall the caller's other streams.  The per-tile
// partials and the completion counter therefore live in one file-scope device
// array of fixed size.
//
// Layout of the array (doubles): one partial per CTA (kNoAllocMaxParts), then
// the completion counter (32 doubles).
// Only the counter must read zero when a call starts: it is zero at module
// load, zeroed again when the address is first resolved on a device, and the
// last CTA of every call puts it back to zero.  The partials are written before
// they are read in every call.  Two calls that overlap
// on one device (different streams, or different host threads without
// ordering) share this array and race.
constexpr int kNoAllocThreads = 256;
constexpr int kNoAllocMaxParts = 148 * 3;  // CTAs
constexpr int kNoAllocPartialDoubles = (int)(sizeof(MomPartial) / sizeof(double));
constexpr size_t kNoAllocCounterOff =
    ((size_t)kNoAllocMaxParts * kNoAllocPartialDoubles + 31) / 32 * 32;
constexpr size_t kNoAllocDoubles = kNoAllocCounterOff + 32;
static_assert(sizeof(MomPartial) % sizeof(double) == 0, "partial is a whole number of doubles");
static_assert((long long)kNoAllocMaxTiles * kTile >= CG_NOALLOC_MAX_PARTICLES,
              "the largest accepted call");
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocDoubles];

cudaError_t noalloc_scratch_address(double** ptr) {
  cudaError_t e = cudaGetSymbolAddress((void**)ptr, g_noalloc_scratch);
  if (e != cudaSuccess) return e;
  return cudaMemset(*ptr + kNoAllocCounterOff, 0, 32 * sizeof(double));
}

__global__ void __launch_bounds__(kNoAllocThreads, 3) k_moments_noalloc(const double* __restrict__ c,
                                                           int64_t stride,
                                                           const uint8_t* __restrict__ surv, int n,
                                                           int steps, double beta_x, double beta_y,
                                                           double* scratch, cg_bunch_moments* out) {
  __shared__ double s_pivot[kNoAllocThreads / 32][6];
  __shared__ MomPartial s_part[kNoAllocThreads / 32];
  __shared__ bool s_last;
  MomPartial* partials = reinterpret_cast<MomPartial*>(scratch);
  unsigned* counter = reinterpret_cast<unsigned*>(scratch + kNoAllocCounterOff);
  const int warp = threadIdx.x >> 5;
  double* pivot = s_pivot[warp];
  MomSums m;
  mom_sums_clear(m);
  bool have = false;
  int i = blockIdx.x * steps * kNoAllocThreads + threadIdx.x;
  // the next step's loads in flight while this one's are added up
  auto load = [&](int at, double (&v)[6]) {
    const bool valid = at < n;
    const bool alive = valid && surv[at] == kAlive;
#pragma unroll
    for (int d = 0; d < 6; ++d) v[d] = valid ? c[d * stride + at] : 0.0;
    return alive;
  };
  double v[6];
  bool next = load(i, v);
#pragma unroll 1
  for (int u = 0; u < steps; ++u) {
    const bool alive = next;
    double w[6];
#pragma unroll
    for (int d = 0; d < 6; ++d) w[d] = v[d];
    if (u + 1 < steps) {
      i += kNoAllocThreads;
      next = load(i, v);
    }
    if (!have) have = mom_pivot(pivot, alive, w);
    if (alive) mom_sums_add<true>(m, w, pivot);
  }
  mom_partial(m, have, pivot, &s_part[warp]);
  __syncthreads();
  if (warp == 0)
    mom_merge_warp<false>(s_part, kNoAllocThreads / 32, 0, 32, pivot, &partials[blockIdx.x]);
  // the last CTA merges
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const MomPartial* total = mom_merge_block<kNoAllocThreads>(partials, (int)gridDim.x);
  if (threadIdx.x != 0) return;
  *counter = 0;
  BunchMomDev s;
  mom_finalize(*total, beta_x, beta_y, c[4 * stride], s);
  // the public record (its transmission is n_alive / n)
  cg_bunch_moments o;
  o.n_alive = (int)s.n_alive;
  o.n_macro = n;
  for (int d = 0; d < 6; ++d) o.mean[d] = s.mean[d];
  for (int d = 0; d < 3; ++d) {
    o.emit[d] = s.emit[d];
    o.eff_emit[d] = s.eff_emit[d];
  }
  o.rms_x = s.rms_x;
  o.rms_y = s.rms_y;
  o.eff_rms_x = s.eff_rms_x;
  o.eff_rms_y = s.eff_rms_y;
  o.bunch_length = s.bunch_length;
  o.energy_spread = s.energy_spread;
  o.z_min = s.z_min;
  o.z_max = s.z_max;
  o.transmission = s.n_alive / (double)n;
  *out = o;
}

// Steps per CTA: enough that at most kNoAllocMaxParts CTAs cover the call, so
// that every CTA of the largest runs at once.
cudaError_t launch_moments_noalloc(const double* c, int64_t stride, const uint8_t* surv, int n,
                                   double beta_x, double beta_y, double* scratch,
                                   cg_bunch_moments* out, cudaStream_t s) {
  if (n < 1 || n > kNoAllocMaxTiles * kTile) return cudaErrorInvalidValue;
  const int all = (n + kNoAllocThreads - 1) / kNoAllocThreads;
  const int steps = (all + kNoAllocMaxParts - 1) / kNoAllocMaxParts;
  k_moments_noalloc<<<(all + steps - 1) / steps, kNoAllocThreads, 0, s>>>(
      c, stride, surv, n, steps, beta_x, beta_y, scratch, out);
  return cudaGetLastError();
}

}  // namespace cg
