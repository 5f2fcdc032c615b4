// Space charge of the electron bunches, per section (runSpaceCharge;
// MPBeam::BeamTransferDueToSpaceChargePIC / ...Analytical, MPBeam.cpp:
// 2565-2583, called before the section map, MPBeam.cpp:1065-1066).
//
// The reference slices each bunch longitudinally (MPBunch::SetSlicedBunchInfo,
// MPBunch.cpp:660-693: nz slices over the survivors' z range, every particle
// in one), and per slice of at least two particles kicks every particle in it
// transversely by the field of the slice's line charge:
//   flag 2: 2.5-D PIC (MPBunch.cpp:887-931, PIC2D.cpp): a mesh of nx x ny
//           nodes from the bunch's rms size and centroid, cloud-in-cell
//           charge, Poisson's equation by 2-D DST-I (FFTW RODFT00) with the
//           five-point Laplacian's eigenvalues, central-difference field,
//           cloud-in-cell interpolation;
//   flag 1: Bassetti-Erskine field of the slice's rms sizes about its
//           centroid (MPBunch.cpp:695-762);
//   flag 3: the linear field of a uniform beam of those sizes (:764-831).
// Every flag ends in the same momentum update (PIC2D.cpp, MPBunch.cpp:740-760).
//
//  k_sc_range    per chunk: the survivors' z range (GetZMinMax, seeded with
//                particle 0) and, for the slice models, the largest |x|, |y|
//                (ordered bit patterns under atomics).  In the turn the PIC
//                takes the range from the moments formed just before.
//  k_sc_geom     per bunch: the slice width, the mesh (PIC2D::Set2DMesh(rms,
//                centroid), PIC2D.cpp), the fixed-point scales.
//  k_sc_count    per chunk: particles per slice in shared memory, then added to
//                the bunch's; slice models: also the sums of x, y, x^2, y^2
//                about the bunch centroid in 64-bit fixed point
//                (order-independent sums under atomics).
//  k_sc_slices   slice models: per slice the centroid, the sizes and the
//                field's constants.
//  k_sc_offsets, k_sc_scatter (PIC): the particles' x, y grouped by slice.
//  k_sc_solve    one CTA per (bunch, slice) (PIC): the slice's cloud-in-cell
//                charge in shared memory (fixed point), the DST-I Poisson
//                solve as two matrix products each way on the FP64 tensor
//                instructions, then the field on the mesh.
//  k_sc_kick     per tile: the field at each particle and the kick.
// Bound by: the passes over the particles by HBM latency and shared-memory
// atomics, the solve by its deposit (the beam's core is a few cells wide) and
// the barriers round four small matrix products, the field models by the FP64
// pipe.  A section of 80 bunches of 20,000, us: PIC 32 x 32 x 33 468 -> 196
// (solve 80, map 47, kick 38, scatter 24, count 13, moments' merge 9, geom 4,
// offsets 3); Bassetti-Erskine slices 373 -> 129.  Before, the transforms were
// plain FP64 dot products, the deposit went through 64-bit shared atomics
// (compare-and-swap loops) from the whole bunch's particles, and the kick
// evaluated w(z) through the general path.  In the solve index arithmetic and
// divisions had cost as much as the products (95 -> 80 us with padded tables,
// two tiles a time and one reciprocal per node); four copies of the charge
// against the deposit's conflicts gained nothing (97).
#include <algorithm>
#include <cuda_runtime.h>

#include "be_field.cuh"
#include "kernels.cuh"
#include "turn_tail.cuh"

namespace cg {

#define SC_FULL 0xffffffffu
constexpr int kScThreads = 256;
constexpr double kEpsilon0 = 8.854187817E-12;  // Global.h:26
constexpr double kElectronMassKg = 9.10938215E-31;

// per-bunch geometry, sc_geom[b * kScGeom + ...]
enum {
  kGZmin = 0, kGDz, kGIDz, kGMx0, kGMy0, kGHx, kGHy, kGIHx, kGIHy, kGIDv,
  kGExp0, kGExp1, kGExp2, kGExp3, kGPx, kGPy
};
static_assert(kGPy + 1 == kScGeom, "geometry record");

__device__ __forceinline__ int sc_fix_exp(double amax, double n) {
  if (!(amax > 0) || isinf(amax)) return 0;
  const int nb = 32 - __clz((int)n);
  return 60 - ilogb(amax) - nb;
}
__device__ __forceinline__ double sc_fix(unsigned long long v, int e) {
  return scalbn((double)(long long)v, -e);
}

// range[4 b ..]: maxima over bunch b, zero between calls: keys (sr_key) of the
// survivors' -z and z (particle 0 not yet in them), bit patterns of |x|, |y|.
template <bool XY>
__global__ void __launch_bounds__(kScThreads) k_sc_range(const double* __restrict__ c, int64_t npad,
                                                         const uint8_t* __restrict__ surv,
                                                         const int4* __restrict__ chunk_loc,
                                                         unsigned long long* range) {
  __shared__ double red[4][kScThreads / 32];
  const int4 l = chunk_loc[blockIdx.x];
  double zmn = INFINITY, zmx = -INFINITY, ax = 0, ay = 0;
  int64_t g = (int64_t)l.y * kTile + threadIdx.x;
  for (int u = 0; u < l.z; ++u, g += kTile) {
    const uint8_t s = surv[g];
    if (s == kPadding) break;  // the tail of the bunch's last tile
    const double z = c[4 * npad + g];
    if (s == kAlive) {
      zmn = fmin(zmn, z);
      zmx = fmax(zmx, z);
    }
    if (XY) {
      ax = fmax(ax, fabs(c[g]));
      ay = fmax(ay, fabs(c[2 * npad + g]));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    zmn = fmin(zmn, __shfl_xor_sync(SC_FULL, zmn, o));
    zmx = fmax(zmx, __shfl_xor_sync(SC_FULL, zmx, o));
    if (XY) {
      ax = fmax(ax, __shfl_xor_sync(SC_FULL, ax, o));
      ay = fmax(ay, __shfl_xor_sync(SC_FULL, ay, o));
    }
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = zmn;
    red[1][threadIdx.x >> 5] = zmx;
    red[2][threadIdx.x >> 5] = ax;
    red[3][threadIdx.x >> 5] = ay;
  }
  __syncthreads();
  if (threadIdx.x >= 4) return;
  double v = red[threadIdx.x][0];
  for (int w = 1; w < kScThreads / 32; ++w)
    v = threadIdx.x == 0 ? fmin(v, red[0][w]) : fmax(v, red[threadIdx.x][w]);
  unsigned long long* r = range + 4 * (size_t)l.x + threadIdx.x;
  if (threadIdx.x < 2) {
    // no survivor leaves the minimum at infinity, the maximum at minus infinity
    if (threadIdx.x == 0 ? v < INFINITY : v > -INFINITY) atomicMax(r, sr_key(threadIdx.x == 0 ? -v : v));
  } else if (XY) atomicMax(r, (unsigned long long)__double_as_longlong(v));
}

// ranges: from `range`; else the moments' (of this section, of the beam as it
// is now: the same numbers).  Clears the counts and, per slice, `per` sums.
__global__ void k_sc_geom(const double* __restrict__ c, int64_t npad,
                          const BunchDev* __restrict__ bunch, const BunchMomDev* __restrict__ mom,
                          ScParams p, unsigned long long* range, bool ranges, double* geom,
                          int* status, int M, int* cnt, unsigned long long* acc, int per) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < M * p.nz) {
    cnt[b] = 0;
    for (int q = 0; q < per; ++q) acc[(size_t)b * per + q] = 0ull;
  }
  if (b >= M) return;
  const BunchDev& Bd = bunch[b];
  if (Bd.n < 1) return;
  const BunchMomDev& m = mom[b];
  double zMin = m.z_min, zMax = m.z_max, rx = 0, ry = 0;
  if (ranges) {
    unsigned long long* r = range + 4 * (size_t)b;
    const double z0 = c[4 * npad + (int64_t)Bd.tile_off * kTile];
    // GetZMinMax (MPBunch.cpp:1883-1884)
    zMin = (r[0] ? fmin(z0, -sr_unkey(r[0])) : z0) - 1.e-6;
    zMax = (r[1] ? fmax(z0, sr_unkey(r[1])) : z0) + 1.e-6;
    rx = __longlong_as_double((long long)r[2]);
    ry = __longlong_as_double((long long)r[3]);
    r[0] = r[1] = r[2] = r[3] = 0ull;
  }
  double* G = geom + (size_t)b * kScGeom;
  // SetSlicedBunchInfo (MPBunch.cpp:670)
  G[kGZmin] = zMin;
  G[kGDz] = (zMax - zMin) / (p.nz - 1);
  G[kGIDz] = 1.0 / G[kGDz];
  const double charge = Bd.q_macro * kElectronCharge / G[kGDz];  // [C/m], MPBunch.cpp:689
  if (p.flag == 2) {
    // PIC2D::Set2DMesh(rmsXY, averXY) (PIC2D.cpp) from the moments of this section
    const double rms[2] = {m.rms_x, m.rms_y}, cen[2] = {m.mean[0], m.mean[2]};
    if (rms[0] == 0 || rms[1] == 0) {
      atomicOr(status, kStatusScMesh);  // MPBunch.cpp:893-897
      G[kGIDv] = 0;
      return;
    }
    double len[2];
    for (int q = 0; q < 2; ++q) len[q] = rms[q] * 2 * p.range;
    const double lmax = len[0] > len[1] ? len[0] : len[1];
    const int n[2] = {p.nx, p.ny};
    double dv = 1.0;
    for (int q = 0; q < 2; ++q) {
      const double w = lmax / (n[q] - 1);
      G[q ? kGHy : kGHx] = w;
      G[q ? kGIHy : kGIHx] = 1.0 / w;
      G[q ? kGMy0 : kGMx0] = cen[q] - lmax / 2;
      dv *= w;
    }
    G[kGIDv] = 1.0 / dv;
    // a deposit is at most charge / dv (weights <= 1)
    G[kGExp0] = sc_fix_exp(charge / dv, Bd.n);
  } else {
    // the sums' pivot: the bunch centroid (zero if there is none)
    const double px = isfinite(m.mean[0]) ? m.mean[0] : 0.0;
    const double py = isfinite(m.mean[2]) ? m.mean[2] : 0.0;
    const double ax = rx + fabs(px), ay = ry + fabs(py);
    G[kGPx] = px;
    G[kGPy] = py;
    G[kGExp0] = sc_fix_exp(ax, Bd.n);
    G[kGExp1] = sc_fix_exp(ay, Bd.n);
    G[kGExp2] = sc_fix_exp(ax * ax, Bd.n);
    G[kGExp3] = sc_fix_exp(ay * ay, Bd.n);
  }
}

// slice of a particle (MPBunch.cpp:679-681); the first for a z that is no
// number (converted, it would index far outside the slices)
__device__ __forceinline__ int sc_slice(double z, const double* G, int nz) {
  const double s = z - G[kGZmin];
  const double t = bin_quotient(s, G[kGDz], G[kGIDz]);
  return !(s > 0) ? 0 : (t < nz - 1 ? (int)t : nz - 1);
}

// mesh cell and cloud-in-cell distances (PIC2D::Set2DRho, PIC2D.cpp: the
// weights times the cell's area); false when the particle is outside the mesh
__device__ __forceinline__ bool sc_cell(double x, double y, const double* G, const ScParams& p,
                                        int* ix, int* iy, double w[4]) {
  const double tx = floor(bin_quotient(x - G[kGMx0], G[kGHx], G[kGIHx]));
  const double ty = floor(bin_quotient(y - G[kGMy0], G[kGHy], G[kGIHy]));
  if (!(tx >= 0 && tx < p.nx - 1 && ty >= 0 && ty < p.ny - 1)) return false;
  *ix = (int)tx;
  *iy = (int)ty;
  const double x1 = fabs(x - (G[kGMx0] + G[kGHx] * (*ix + 1))), x0 = fabs(x - (G[kGMx0] + G[kGHx] * *ix));
  const double y1 = fabs(y - (G[kGMy0] + G[kGHy] * (*iy + 1))), y0 = fabs(y - (G[kGMy0] + G[kGHy] * *iy));
  w[0] = x1 * y1;
  w[1] = x0 * y1;
  w[2] = x1 * y0;
  w[3] = x0 * y0;
  return true;
}

// Slices up to which a CTA keeps its counts (and the models' sums) in shared
// memory; beyond, it adds to the bunch's directly.
constexpr int kScSharedSlices = 1024;

template <bool PIC>
__global__ void __launch_bounds__(kScThreads) k_sc_count(const double* __restrict__ c, int64_t npad,
                                                         const uint8_t* __restrict__ surv,
                                                         const int4* __restrict__ chunk_loc,
                                                         ScParams p, const double* __restrict__ geom,
                                                         int* cnt, unsigned long long* acc) {
  extern __shared__ unsigned s_sum[];  // nz counts; models: then 4 x (lo, hi) x nz
  const int4 l = chunk_loc[blockIdx.x];
  const double* G = geom + (size_t)l.x * kScGeom;
  if (PIC && G[kGIDv] == 0) return;
  const int nz = p.nz;
  const bool shared = nz <= kScSharedSlices;
  if (shared) {
    for (int i = threadIdx.x; i < nz * (PIC ? 1 : 9); i += kScThreads) s_sum[i] = 0u;
    __syncthreads();
  }
  const size_t b0 = (size_t)l.x * nz;
  Pow2 f[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) f[q] = PIC ? Pow2{0, 0} : pow2_split((int)G[kGExp0 + q]);
  int64_t g = (int64_t)l.y * kTile + threadIdx.x;
  for (int u = 0; u < l.z; ++u, g += kTile) {
    const uint8_t sv = surv[g];
    const double z = c[4 * npad + g];
    if (sv == kPadding) break;
    const int s = sc_slice(z, G, nz);
    if (shared) atomicAdd(&s_sum[s], 1u);
    else atomicAdd(&cnt[b0 + s], 1);
    if (!PIC) {
      const double dx = c[g] - G[kGPx], dy = c[2 * npad + g] - G[kGPy];
      const double v[4] = {dx, dy, dx * dx, dy * dy};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const long long t = __double2ll_rn(pow2_scale(v[q], f[q]));
        if (shared) add64_split(&s_sum[(1 + 2 * q) * nz + s], &s_sum[(2 + 2 * q) * nz + s], t);
        else atomicAdd(&acc[(b0 + s) * 4 + q], (unsigned long long)t);
      }
    }
  }
  if (!shared) return;
  __syncthreads();
  for (int s = threadIdx.x; s < nz; s += kScThreads) {
    if (!s_sum[s]) continue;
    atomicAdd(&cnt[b0 + s], (int)s_sum[s]);
    if (!PIC)
      for (int q = 0; q < 4; ++q)
        atomicAdd(&acc[(b0 + s) * 4 + q],
                  (unsigned long long)s_sum[(2 + 2 * q) * nz + s] << 32 | s_sum[(1 + 2 * q) * nz + s]);
  }
}

// Slice models: one slice as the kick reads it.
struct ScSlice {
  double cx, cy, rx, ry;  // centroid, sizes
  double lambda;          // line charge over pi epsilon0
  KickConst k;            // flag 1: the field's constants, in the frame of the larger axis
};

__global__ void k_sc_slices(ScParams p, const BunchDev* __restrict__ bunch,
                            const double* __restrict__ geom, const int* __restrict__ cnt,
                            const unsigned long long* __restrict__ acc, ScSlice* slices, int M) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= M * p.nz) return;
  const int b = i / p.nz, n = cnt[i];
  if (n < 2) return;
  const double* G = geom + (size_t)b * kScGeom;
  const unsigned long long* A = acc + 4 * (size_t)i;
  const double mx = sc_fix(A[0], (int)G[kGExp0]) / n, my = sc_fix(A[1], (int)G[kGExp1]) / n;
  ScSlice s;
  s.cx = G[kGPx] + mx;
  s.cy = G[kGPy] + my;
  s.rx = sqrt(fmax(sc_fix(A[2], (int)G[kGExp2]) / n - mx * mx, 0.0));
  s.ry = sqrt(fmax(sc_fix(A[3], (int)G[kGExp3]) / n - my * my, 0.0));
  s.lambda = n * (bunch[b].q_macro * kElectronCharge / G[kGDz]) / kPi / kEpsilon0;  // n charge: [C/m]
  CloudRec r;
  r.coeff = -0.5 * s.lambda;
  r.rms_x = s.rx;
  r.rms_y = s.ry;
  r.aver_x = s.cx;
  r.aver_y = s.cy;
  r.count = n;
  s.k = kick_const(r, field_prep(s.rx, s.ry));
  slices[i] = s;
}

// PIC: each bunch's particles grouped by slice (a counting sort: the slices'
// starts, then every particle's x, y at its slice's cursor), so that one CTA
// per slice deposits its own particles in shared memory.  One warp per bunch.
__global__ void k_sc_offsets(const BunchDev* __restrict__ bunch, int nz, const int* __restrict__ cnt,
                             int* start, int* cursor) {
  const int b = blockIdx.x, lane = threadIdx.x;
  int base = bunch[b].tile_off * kTile;
  for (int s0 = 0; s0 < nz; s0 += 32) {
    const int s = s0 + lane, n = s < nz ? cnt[(size_t)b * nz + s] : 0;
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(SC_FULL, inc, o);
      if (lane >= o) inc += t;
    }
    if (s < nz) start[(size_t)b * nz + s] = cursor[(size_t)b * nz + s] = base + inc - n;
    base += __shfl_sync(SC_FULL, inc, 31);
  }
}

__global__ void __launch_bounds__(kScThreads) k_sc_scatter(const double* __restrict__ c, int64_t npad,
                                                           const uint8_t* __restrict__ surv,
                                                           const int4* __restrict__ chunk_loc,
                                                           ScParams p,
                                                           const double* __restrict__ geom,
                                                           int* cursor, double2* xy) {
  extern __shared__ unsigned s_sum[];  // nz counts, then nz first places
  const int4 l = chunk_loc[blockIdx.x];
  const double* G = geom + (size_t)l.x * kScGeom;
  if (G[kGIDv] == 0) return;
  const int nz = p.nz;
  const bool shared = nz <= kScSharedSlices;
  const size_t b0 = (size_t)l.x * nz;
  const int64_t g0 = (int64_t)l.y * kTile + threadIdx.x;
  unsigned rank[kMaxChunkTiles];
  int slot[kMaxChunkTiles];
  if (shared) {
    // the chunk's places in each slice with one global atomic per slice
    for (int i = threadIdx.x; i < nz; i += kScThreads) s_sum[i] = 0u;
    __syncthreads();
    for (int u0 = 0; u0 < l.z; u0 += kMaxChunkTiles) {
      const int nu = min(kMaxChunkTiles, l.z - u0);
#pragma unroll
      for (int u = 0; u < kMaxChunkTiles; ++u) {
        const int64_t g = g0 + (int64_t)(u0 + u) * kTile;
        if (u >= nu) break;
        const uint8_t sv = surv[g];
        const double z = c[4 * npad + g];
        slot[u] = sv != kPadding ? sc_slice(z, G, nz) : -1;
        if (slot[u] >= 0) rank[u] = atomicAdd(&s_sum[slot[u]], 1u);
      }
      __syncthreads();
      for (int s = threadIdx.x; s < nz; s += kScThreads) {
        s_sum[nz + s] = s_sum[s] ? (unsigned)atomicAdd(&cursor[b0 + s], (int)s_sum[s]) : 0u;
        s_sum[s] = 0u;
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < kMaxChunkTiles; ++u) {
        const int64_t g = g0 + (int64_t)(u0 + u) * kTile;
        if (u >= nu) break;
        const double2 v = make_double2(c[g], c[2 * npad + g]);
        if (slot[u] >= 0) xy[s_sum[nz + slot[u]] + rank[u]] = v;
      }
      __syncthreads();
    }
  } else {
    for (int u = 0; u < l.z; ++u) {
      const int64_t g = g0 + (int64_t)u * kTile;
      if (surv[g] != kPadding)
        xy[atomicAdd(&cursor[b0 + sc_slice(c[4 * npad + g], G, nz)], 1)] = make_double2(c[g], c[2 * npad + g]);
    }
  }
}

// D = A B on the FP64 tensor instructions (m8n8k4): one or two neighbouring
// 8 x 8 tiles of a row of the product of A (rows, K) and B (K, columns), both
// row by row in shared memory with a row stride of 4 or 12 modulo 16 doubles
// (no bank conflicts).  Lane l gets the elements (l / 4, 2 (l % 4)) and the
// next.  Two tiles share A's loads, and one waits while the other multiplies.
__device__ __forceinline__ void sc_mma(double a, double b, double (&d)[2]) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}
__device__ __forceinline__ void sc_mma_tiles(const double* A, int lda, const double* B, int ldb, int K,
                                             bool two, double (&d)[2][2]) {
  const int lane = threadIdx.x & 31;
  const double* a = A + (lane >> 2) * lda + (lane & 3);
  const double* b = B + (lane & 3) * ldb + (lane >> 2);
  d[0][0] = d[0][1] = d[1][0] = d[1][1] = 0.0;
  const int step = 4 * ldb;
  if (two) {
#pragma unroll 2
    for (int k = 0; k < K; k += 8, a += 8, b += 2 * step) {  // K: whole tiles
      const double a0 = a[0], a1 = a[4], b0 = b[0], c0 = b[8], b1 = b[step], c1 = b[step + 8];
      sc_mma(a0, b0, d[0]);
      sc_mma(a0, c0, d[1]);
      sc_mma(a1, b1, d[0]);
      sc_mma(a1, c1, d[1]);
    }
  } else {
    for (int k = 0; k < K; k += 4, a += 4, b += step) sc_mma(a[0], b[0], d[0]);
  }
}

// One CTA per (bunch, slice): PIC2D::Set2DPhi and Set2DEField (PIC2D.cpp).
// The 2-D DST-I (RODFT00, Y_k = 2 sum_j X_j sin(pi (j + 1)(k + 1) / (n + 1))
// along each axis) as S_x R S_y^T in shared memory; sx, sy hold 2 sin(...),
// the mesh padded with zeros to whole 8 x 8 tiles.
__global__ void __launch_bounds__(kScThreads) k_sc_solve(ScParams p, const BunchDev* __restrict__ bunch,
                                                         const double* __restrict__ geom,
                                                         const int* __restrict__ cnt,
                                                         const int* __restrict__ start,
                                                         const double2* __restrict__ xy,
                                                         const double* __restrict__ sxy,
                                                         double* field) {
  extern __shared__ double sm[];
  const int nx = p.nx, ny = p.ny, N = nx * ny;
  const int b = blockIdx.x / p.nz;
  const size_t bs = blockIdx.x;
  const double* G = geom + (size_t)b * kScGeom;
  const int n = cnt[bs];
  if (n < 2 || G[kGIDv] == 0) return;  // a skipped slice (MPBunch.cpp:916)
  const int px = sc_pad(nx), py = sc_pad(ny), lx = sc_stride(px), ly = sc_stride(py);
  double* R = sm;                // px x ly
  double* T = R + px * ly;       // px x ly
  double* Sx = T + px * ly;      // px x lx
  double* Sy = Sx + px * lx;     // py x ly
  unsigned* lo = reinterpret_cast<unsigned*>(T);  // the fixed-point charge, in T's place
  unsigned* hi = lo + N;
  const int e = (int)G[kGExp0];
  for (int t = threadIdx.x; t < 2 * N; t += kScThreads) lo[t] = 0u;
  // Sx and Sy one after the other, here and in the table
  for (int t = threadIdx.x; t < (px * lx + py * ly) / 2; t += kScThreads)
    reinterpret_cast<double2*>(Sx)[t] = __ldg(reinterpret_cast<const double2*>(sxy) + t);
  __syncthreads();
  // PIC2D::Set2DRho (PIC2D.cpp): cloud-in-cell charge [C/m^3] of the slice's
  // particles, in 64-bit fixed point (order-independent)
  const double charge = bunch[b].q_macro * kElectronCharge / G[kGDz];
  const double unit = scalbn(charge * G[kGIDv] * G[kGIDv], e);
  const double2* L = xy + start[bs];
  for (int t = threadIdx.x; t < n; t += kScThreads) {
    const double2 v = L[t];
    int ix, iy;
    double w[4];
    if (!sc_cell(v.x, v.y, G, p, &ix, &iy, w)) continue;
    const int node[4] = {ix * ny + iy, (ix + 1) * ny + iy, ix * ny + iy + 1, (ix + 1) * ny + iy + 1};
#pragma unroll
    for (int j = 0; j < 4; ++j) add64_split(&lo[node[j]], &hi[node[j]], __double2ll_rn(w[j] * unit));
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Pow2 back = pow2_split(-e);
  for (int i = warp; i < px; i += kScThreads / 32)
    for (int j = lane; j < ly; j += 32)
      R[i * ly + j] = i < nx && j < ny
                          ? pow2_scale((double)(long long)((unsigned long long)hi[i * ny + j] << 32 |
                                                           lo[i * ny + j]), back)
                          : 0.0;
  __syncthreads();
  const double hx = G[kGHx], hy = G[kGHy];
  const double* __restrict__ eig = sxy + px * lx + py * ly;
  const int tx = px / 8, ty = py / 8, half = (ty + 1) / 2;
  const double sx2 = 2 / hx, sy2 = 2 / hy, norm = 1.0 / (4.0 * (nx + 1) * (ny + 1));
  for (int pass = 0; pass < 2; ++pass) {
    double d[2][2];
    for (int q = warp; q < tx * half; q += kScThreads / 32) {  // T = Sx R (along x)
      const int i = q / half * 8, j = q % half * 16;
      const bool two = j + 8 < py;
      sc_mma_tiles(Sx + i * lx, lx, R + j, ly, px, two, d);
      double* o = T + (i + (lane >> 2)) * ly + j + 2 * (lane & 3);
      *reinterpret_cast<double2*>(o) = make_double2(d[0][0], d[0][1]);
      if (two) *reinterpret_cast<double2*>(o + 8) = make_double2(d[1][0], d[1][1]);
    }
    __syncthreads();
    for (int q = warp; q < tx * half; q += kScThreads / 32) {  // R = T Sy^T (along y; Sy is symmetric)
      const int i = q / half * 8, j = q % half * 16;
      const bool two = j + 8 < py;
      sc_mma_tiles(T + i * ly, ly, Sy + j, ly, py, two, d);
      const int k = i + (lane >> 2);
      // the Laplacian's eigenvalue (PIC2D.cpp Set2DPhi): out / K / Epsilon,
      // with the sines of pi / 2 (k + 1) / (n + 1) from the table
      const double ax = k < nx ? sx2 * eig[k] : 0.0;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (u >= 2 && !two) break;
        const int m = j + 8 * (u >> 1) + 2 * (lane & 3) + (u & 1);
        double v = 0.0;
        if (k < nx && m < ny) {
          const double ay = pass == 0 ? sy2 * eig[nx + m] : 0.0;
          v = d[u >> 1][u & 1] *
              (pass == 0 ? recip_newton(fma(ax, ax, ay * ay)) * (1.0 / kEpsilon0) : norm);  // phi [V]
        }
        R[k * ly + m] = v;
      }
    }
    __syncthreads();
  }
  // Set2DEField: central differences, zero potential beyond the mesh
  double* F = field + bs * 2 * N;
  const double fx = -0.5 / hx, fy = -0.5 / hy;
  for (int i = warp; i < nx; i += kScThreads / 32)
    for (int j = lane; j < ny; j += 32) {
      const double x1 = i == 0 ? 0 : R[(i - 1) * ly + j], x2 = i == nx - 1 ? 0 : R[(i + 1) * ly + j];
      const double y1 = j == 0 ? 0 : R[i * ly + j - 1], y2 = j == ny - 1 ? 0 : R[i * ly + j + 1];
      reinterpret_cast<double2*>(F)[i * ny + j] = make_double2((x2 - x1) * fx, (y2 - y1) * fy);
    }
}

// A point beyond the series' range or a round slice, out of line.
__device__ __noinline__ void sc_field_any(const ScSlice& s, double posx, double posy, double* fx,
                                          double* fy) {
  if ((s.rx - s.ry) / s.ry > 1.e-4) bassetti_erskine(posx, posy, s.rx, s.ry, fx, fy);
  else if ((s.rx - s.ry) / s.ry < -1.e-4) bassetti_erskine(posy, posx, s.ry, s.rx, fy, fx);
  else gaussian_round_field(posx, posy, s.rx, fx, fy);
}

// The kick (PIC2D::SetPartSCField / UpdateTransverseMomentum, PIC2D.cpp;
// MPBunch.cpp:713-760 and 781-829); its total momentum p is formed from
// (delta, y, px) as there, and E / gamma^2 e ds / (beta c) / (m p c) is
// evaluated as E e ds / (m c^2) / (gamma p^2).
template <int FLAG>
__global__ void __launch_bounds__(kTile) k_sc_kick(double* __restrict__ c, int64_t npad,
                                                   const uint8_t* __restrict__ surv,
                                                   const int* __restrict__ tile_bunch, ScParams p,
                                                   const double* __restrict__ geom,
                                                   const int* __restrict__ cnt,
                                                   const ScSlice* __restrict__ slices,
                                                   const double* __restrict__ field, double ds) {
  const int b = tile_bunch[blockIdx.x];
  const int64_t g = (int64_t)blockIdx.x * kTile + threadIdx.x;
  // every load that waits for no other first, but for the model that the FP64
  // pipe bounds (padding slots hold numbers)
  const uint8_t sv = surv[g];
  if (FLAG == 1 && sv == kPadding) return;
  const double z = c[4 * npad + g], x = c[g], y = c[2 * npad + g];
  const double px0 = c[npad + g], py0 = c[3 * npad + g], dp = c[5 * npad + g];
  const double* G = geom + (size_t)b * kScGeom;
  if (sv == kPadding || (FLAG == 2 && G[kGIDv] == 0)) return;
  const int s = sc_slice(z, G, p.nz);
  const size_t bs = (size_t)b * p.nz + s;
  const int in_slice = cnt[bs];
  if (FLAG == 1 && in_slice < 2) return;
  double ex = 0, ey = 0;
  if (FLAG == 2) {
    int ix, iy;
    double w[4];
    if (sc_cell(x, y, G, p, &ix, &iy, w)) {
      const double2* F = reinterpret_cast<const double2*>(field) + bs * p.nx * p.ny;
      const int n0 = ix * p.ny + iy;
      const double2 f0 = F[n0], f1 = F[n0 + p.ny], f2 = F[n0 + 1], f3 = F[n0 + p.ny + 1];
      ex = (f0.x * w[0] + f1.x * w[1] + f2.x * w[2] + f3.x * w[3]) * G[kGIDv];
      ey = (f0.y * w[0] + f1.y * w[1] + f2.y * w[2] + f3.y * w[3]) * G[kGIDv];
    }
  }
  if (in_slice < 2) return;  // MPBunch.cpp:916 (the mesh's loads do not wait for it)
  if (FLAG == 1) {
    const ScSlice& S = slices[bs];
    const KickConst& k = S.k;
    const bool sw = k.mode == 1;
    const double da = (sw ? y : x) - k.ma, db = (sw ? x : y) - k.mb;
    const double aa = fabs(da), ab = fabs(db);
    const double zr[2] = {aa * k.s0, aa * k.sa1}, zi[2] = {ab * k.s0, ab * k.sb1};
    constexpr int kHi21 = 0x40350000;  // |z| < 30 in both series (see ion_kick_particle)
    if (k.mode != 2 && __double2hiint(zr[0]) < kHi21 && __double2hiint(zi[1]) < kHi21) {
      const double ua = aa * k.ga, ub = ab * k.gb;
      const double gs = exp_neg(0.5 * fma(ua, ua, ub * ub));
      cplx w[2];
      w_weideman_fast<2>(zr, zi, w);
      const double fa = flip_sign(k.ck * fma(-gs, w[1].im, w[0].im), da);
      const double fb = flip_sign(k.ck * fma(-gs, w[1].re, w[0].re), db);
      ex = sw ? fb : fa;
      ey = sw ? fa : fb;
    } else {
      double fx, fy;
      sc_field_any(S, x - S.cx, y - S.cy, &fx, &fy);
      ex = -0.5 * S.lambda * fx;
      ey = -0.5 * S.lambda * fy;
    }
  } else if (FLAG == 3) {
    const ScSlice& S = slices[bs];
    const double q = S.lambda / (S.rx + S.ry);
    ex = q * ((x - S.cx) / S.rx);
    ey = q * ((y - S.cy) / S.ry);
  }
  const double pz = (1 + dp) * p.p0;
  const double tpx = pz * y, tpy = pz * px0;
  const double p2 = pz * pz + tpx * tpx + tpy * tpy;
  const double f = kElectronCharge * ds / (kElectronMassKg * kCLight * kCLight) / (sqrt(1 + p2) * p2);
  c[npad + g] = px0 + ex * f;
  c[3 * npad + g] = py0 + ey * f;
}

// this translation unit's copy of the w(z) table (faddeeva.cuh keeps one
// __constant__ copy per unit)
cudaError_t upload_weideman_table_sc() {
  return cudaMemcpyToSymbol(c_weideman, &h_weideman, sizeof(WeidemanTable));
}

size_t sc_solve_smem(const ScParams& p) {
  const size_t px = sc_pad(p.nx), py = sc_pad(p.ny);
  return sizeof(double) * (2 * px * (py + 4) + px * (px + 4) + py * (py + 4));
}

size_t sc_slice_bytes() { return sizeof(ScSlice); }

cudaError_t prepare_sc(const ScParams& p) {
  if (p.flag != 2) return cudaSuccess;
  return cudaFuncSetAttribute(k_sc_solve, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)sc_solve_smem(p));
}

cudaError_t launch_space_charge(Handle& h, int k, bool have_range) {
  const ScParams& p = h.sc;
  const DeviceBufs& d = h.d;
  const cudaStream_t st = h.stream;
  const bool pic = p.flag == 2;
  const int slices = h.M * p.nz;
  const size_t shared = p.nz <= kScSharedSlices ? sizeof(unsigned) * p.nz : 0;
  if (h.n_chunks < 1) return cudaSuccess;
  ScSlice* sl = reinterpret_cast<ScSlice*>(d.sc_slices);
  double2* xy = reinterpret_cast<double2*>(d.sc_xy);
  const bool ranges = !(pic && have_range);
  if (ranges)
    (pic ? k_sc_range<false> : k_sc_range<true>)<<<h.n_chunks, kScThreads, 0, st>>>(
        d.c, h.npad, d.surv, d.chunk_loc, d.sc_range);
  k_sc_geom<<<(slices + 127) / 128, 128, 0, st>>>(d.c, h.npad, d.bunch, d.mom, p, d.sc_range, ranges,
                                                  d.sc_geom, d.status, h.M, d.sc_cnt, d.sc_acc,
                                                  pic ? 0 : 4);
  (pic ? k_sc_count<true> : k_sc_count<false>)<<<h.n_chunks, kScThreads, shared * (pic ? 1 : 9), st>>>(
      d.c, h.npad, d.surv, d.chunk_loc, p, d.sc_geom, d.sc_cnt, d.sc_acc);
  if (pic) {
    k_sc_offsets<<<h.M, 32, 0, st>>>(d.bunch, p.nz, d.sc_cnt, d.sc_start, d.sc_cursor);
    k_sc_scatter<<<h.n_chunks, kScThreads, 2 * shared, st>>>(d.c, h.npad, d.surv, d.chunk_loc, p,
                                                             d.sc_geom, d.sc_cursor, xy);
    k_sc_solve<<<slices, kScThreads, sc_solve_smem(p), st>>>(p, d.bunch, d.sc_geom, d.sc_cnt,
                                                             d.sc_start, xy, d.sc_sin, d.sc_field);
  } else {
    k_sc_slices<<<(slices + 127) / 128, 128, 0, st>>>(p, d.bunch, d.sc_geom, d.sc_cnt, d.sc_acc, sl,
                                                      h.M);
  }
  auto kick = pic ? k_sc_kick<2> : p.flag == 1 ? k_sc_kick<1> : k_sc_kick<3>;
  kick<<<h.n_tiles, kTile, 0, st>>>(d.c, h.npad, d.surv, d.tile_bunch, p, d.sc_geom, d.sc_cnt, sl,
                                    d.sc_field, h.sections[k].length);
  return cudaGetLastError();
}

}  // namespace cg
