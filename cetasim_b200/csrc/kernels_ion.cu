// Ion chain of one interaction point (MPBeam::SSBeamIonEffectOneInteraction
// Point, MPBeam.cpp:2585-2611) as independent ion trajectories.
//
// In the reference, bunch j of the train meets the cloud the previous bunches
// left behind: macro-ions are born (LIP::IonGenerator, LIP.cpp:985-1019) and
// appended (IonsUpdate, :1021-1051), the cloud's moments are taken
// (IonRMSCal, :1113-1155) for the electron-side kick, every ion is kicked by
// the field of bunch j (MPBunch.cpp:1111-1157), drifts over the gap to the
// next bunch and is erased beyond the loss bound (IonTransferDueToBunch,
// LIP.cpp:1158-1211).  The ions never act on one another: an ion's motion
// depends only on the bunches it meets, whose centroids and sizes are fixed
// for the call, and the loss bound min(aperture, boundary * max sigma) is
// fixed for the call too (MPBeam.cpp:2257).  So the chain is a set of
// independent trajectories - the ions already in the cloud, then the ions
// born at bunch j, in the reference's order - and the only quantities that
// couple them are the cloud moments each bunch sees, which are per-step sums
// over the ions alive at that step.
//
// Four kernels per IP:
//   k_ion_prep    per bunch: loss bounds, birth positions (Philox, attempts in
//                 order), field constants, coefficients;
//   k_ion_walk    each CTA walks 16 to 128 trajectories (two lanes per ion, one
//                 for w(z1) and one for w(z2), or one lane for both) through all
//                 bunches without a barrier per bunch, and writes per-step partial
//                 sums (count, sum x, y, x^2, y^2) every kWin bunches;
//   k_ion_records one warp per step: sums in a fixed order -> cloud centroid and
//                 rms -> the record the electron kick reads;
//   k_ion_compact stable compaction of the survivors into the cloud (birth
//                 order, as the reference's erase keeps it) and the cloud state.
// The walk and the records also run as consecutive segments of bunch steps.
// The critical path is one field evaluation per bunch passage of the longest
// trajectory, instead of a block-synchronised cloud pass per bunch.
#include <cuda_runtime.h>
#include <algorithm>
#include "kernels.cuh"

namespace cg {

#define FULL_MASK 0xffffffffu

// The walk's CTA shape: IONS trajectories per block (16, 32 or 64) with two
// lanes each, or 2 IONS with one lane each (see k_ion_walk).
constexpr int kWin = 16;                       // steps per shared-memory window
// Trajectories of one species above which one lane walks a whole ion: at two
// lanes per ion the 592 sub-partitions then hold two warps each, which take
// 870 cycles a step together, as much as one warp of whole ions (2415 cycles
// for four); below, the shorter chain of the two lanes wins.
constexpr int64_t kWalkWide = 148 * 4 * 32;
constexpr int kPrepThreads = 128;
constexpr int kRecThreads = 256;
constexpr int kRecChunk = 2048;                // steps per shared-memory chunk of the carry
constexpr int kCompactThreads = 1024;

__device__ __forceinline__ void warp_max2(double& a, double& b) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a = fmax(a, __shfl_xor_sync(FULL_MASK, a, o));
    b = fmax(b, __shfl_xor_sync(FULL_MASK, b, o));
  }
}

// Loss bounds, births and per-bunch constants for one IP: block 0 also takes
// the loss bounds; one warp per (species, bunch) the rest.
__global__ void __launch_bounds__(kPrepThreads) k_ion_prep(ChainParams cp, ChainSection cs,
                                                         const BunchDev* __restrict__ bunch,
                                                         const BunchMomDev* __restrict__ mom,
                                                         IonWalk w, int* status,
                                                         const int* __restrict__ d_turn, int k) {
  __shared__ double s_mx[kPrepThreads / 32], s_my[kPrepThreads / 32];
  const int tid = threadIdx.x, M = cp.n_bunches, NM = cp.macro_per_ip, P = cp.n_species;
  if (blockIdx.x == 0) {
    // MPGetBeamInfo: bunchSizeXMax / YMax (MPBeam.cpp:2175-2186); the maximum
    // does not depend on the order of comparison
    double mx = -INFINITY, my = -INFINITY;
    for (int j = tid; j < M; j += kPrepThreads) {
      mx = fmax(mx, mom[j].rms_x);
      my = fmax(my, mom[j].rms_y);
    }
    warp_max2(mx, my);
    if ((tid & 31) == 0) {
      s_mx[tid >> 5] = mx;
      s_my[tid >> 5] = my;
    }
    __syncthreads();
    if (tid == 0) {
      for (int u = 1; u < kPrepThreads / 32; ++u) {
        mx = fmax(mx, s_mx[u]);
        my = fmax(my, s_my[u]);
      }
      const double lbx = cp.loss_boundary * mx, lby = cp.loss_boundary * my;
      w.bound[0] = cs.aperture_x > lbx ? lbx : cs.aperture_x;  // LIP.cpp:1172-1181
      w.bound[1] = cs.aperture_y > lby ? lby : cs.aperture_y;
    }
  }
  // one warp per (species, bunch): w = p * M + j
  const int lane = tid & 31;
  const int wid = (int)(blockIdx.x * (kPrepThreads / 32)) + (tid >> 5);
  if (wid >= M * P) return;
  const int j = wid % M, p = wid / M;
  const double mx = mom[j].mean[0], my = mom[j].mean[2];
  const double sx = mom[j].rms_x, sy = mom[j].rms_y;
  const double ne = bunch[j].ne;
  if (p == 0 && lane == 0) {
    w.prep[j] = field_prep(sx, sy);
    w.bunch[3 * j + 0] = mx;
    w.bunch[3 * j + 1] = my;
    // drift time to the next bunch: gap * C/h / c (LIP.cpp:1172-1173)
    w.bunch[3 * j + 2] = cp.circ_ring / cp.harmonics * bunch[j].gap / kCLight;
  }
  if (lane == 0) {
    // LIP::GetIonNumberPerInterAction (LIP.cpp:974-982) and the macro-ion
    // charge of IonGenerator (LIP.cpp:985-995)
    const double press_p = cp.gas_percent[p] * cs.pressure;
    const double line_density = cp.cross_section[p] * press_p / cs.temperature / kBoltzmann * ne;
    const double ion_number = line_density * cs.length;
    w.spec[2 * ((size_t)p * M + j) + 0] = ion_number / NM;
    // ion-side coefficient 2 N_e r_e (m_e / m_ion A) c (MPBunch.cpp:1117)
    w.spec[2 * ((size_t)p * M + j) + 1] =
        2.0 * ne * kElecClassicRadius * kElectronMassEV / kIonMassEV / cp.mass_number[p] * kCLight;
  }
  // births: Gaussian around the bunch centroid with the bunch sizes,
  // rejected beyond r^2 > 4 (LIP.cpp:1000-1016); attempt a of bunch j, IP k,
  // species p draws Philox({a, j, turn, 8k + p}).  The warp tries 32
  // attempts at once and keeps the accepted ones in attempt order, which are
  // the births the sequential loop makes.
  const uint32_t turn = (uint32_t)(*d_turn);
  const uint32_t k0 = (uint32_t)cp.seed, k1 = (uint32_t)(cp.seed >> 32) ^ kStreamIonBirth;
  double* out = w.births + 2 * ((size_t)p * M + j) * NM;
  int got = 0;
  for (uint32_t a0 = 0; got < NM; a0 += 32) {
    if (a0 >= (1u << 20)) {  // a degenerate bunch size would reject forever
      if (lane == 0) atomicOr(status, kStatusIonBirth);
      for (int q = got + lane; q < NM; q += 32) out[2 * q] = out[2 * q + 1] = 0.0;
      break;
    }
    u32x4 ctr = {{a0 + (uint32_t)lane, (uint32_t)j, turn, (uint32_t)(k * CG_MAX_SPECIES + p)}};
    double g0, g1;
    normal2(philox4x32_10(ctr, k0, k1), &g0, &g1);
    const double tx = mx + sx * g0, ty = my + sy * g1;
    const double ax = (tx - mx) / sx, ay = (ty - my) / sy;
    const bool ok = !(ax * ax + ay * ay > 4.E0);
    const unsigned acc = __ballot_sync(FULL_MASK, ok);
    const int slot = got + __popc(acc & ((1u << lane) - 1u));
    if (ok && slot < NM) {
      out[2 * slot] = tx;
      out[2 * slot + 1] = ty;
    }
    got += __popc(acc);
  }
}

// One bunch passage as every ion of a window step sees it, in the frame of
// the bunch's axes (a the larger one): the centroid, the scales of w(z1),
// w(z2) and of the Gaussian factor, and the ion-side coefficient.
struct WalkStep {
  double ma, mb;        // centroid
  double sa[2], sb[2];  // z1, z2 = (|da| sa, |db| sb)
  double ga, gb;        // 1/sigma_a, 1/sigma_b
  double c1;            // coefficient times -sqrt(pi)/sigma
  double ci;            // coefficient
  double dt;            // drift time to the next bunch
  int mode;             // FieldPrep::mode: 1 = a is y
};

__device__ __forceinline__ WalkStep walk_step_of(const FieldPrep& f, const double* bunch, double ci) {
  WalkStep s;
  const bool sw = f.mode == 1;
  s.ma = sw ? bunch[1] : bunch[0];
  s.mb = sw ? bunch[0] : bunch[1];
  s.sa[0] = s.sb[0] = f.isig;
  s.sa[1] = f.r * f.isig;
  s.sb[1] = f.isig * f.ir;
  s.ga = f.ia;
  s.gb = f.ib;
  s.c1 = f.coeff * ci;
  s.ci = ci;
  s.dt = bunch[2];
  s.mode = f.mode;
  return s;
}

// What a window's steps may assume (bits, all steps of the window together).
enum : int {
  kWinFlip = 1,  // some bunch has a = y
  kWinStay = 2,  // some bunch has a = x
  kWinSlow = 4,  // a round bunch, or an ion within the loss bounds may see |z| >= 30
};
// For an ion with |x| <= bx, |y| <= by.
__device__ __forceinline__ int walk_step_flags(const WalkStep& s, double bx, double by) {
  if (s.mode == 2) return kWinSlow;
  const double a = (s.mode == 1 ? by : bx) + fabs(s.ma), b = (s.mode == 1 ? bx : by) + fabs(s.mb);
  const double ar = a * fmax(s.sa[0], s.sa[1]), bi = b * fmax(s.sb[0], s.sb[1]);
  return (s.mode == 1 ? kWinFlip : kWinStay) | (fma(ar, ar, bi * bi) < 900.0 ? 0 : kWinSlow);
}

// An ion in the frame (a, b).
struct IonState {
  double a, b, va, vb;
  double ka, kb;  // the last bunch's velocity kick (ionAccumuFx/Fy)
  bool alive;
  __device__ __forceinline__ void flip() {
    double t = a; a = b; b = t;
    t = va; va = vb; vb = t;
    t = ka; ka = kb; kb = t;
  }
};

// The constants of one step in registers: PAIR: of this lane's w(z) alone.
template <bool PAIR>
struct StepRegs {
  double ma, mb, sa[2], sb[2], ga, gb, c1, dt;
};
template <bool PAIR>
__device__ __forceinline__ StepRegs<PAIR> step_regs(const WalkStep& s, int sub) {
  StepRegs<PAIR> r;
  r.ma = s.ma;
  r.mb = s.mb;
  r.sa[0] = s.sa[sub];
  r.sb[0] = s.sb[sub];
  if (!PAIR) {
    r.sa[1] = s.sa[1];
    r.sb[1] = s.sb[1];
  }
  r.ga = s.ga;
  r.gb = s.gb;
  r.c1 = s.c1;
  r.dt = s.dt;
  return r;
}

// Velocity kick, drift and loss test (LIP::IonTransferDueToBunch).
__device__ __forceinline__ void walk_move(double fa, double fb, double dt, bool active, double ba,
                                          double bb, IonState& q) {
  if (active) {
    q.ka = fa;
    q.kb = fb;
    q.va += fa;
    q.vb += fb;
    q.a += q.va * dt;
    q.b += q.vb * dt;
    q.alive = !(fabs(q.a) > ba || fabs(q.b) > bb);
  }
}

// The ion side of MPBunch::SSIonBunchInteraction for one ion and one bunch
// that is not round, all |z| < 30.  PAIR: two lanes per ion, lane `sub`
// evaluates w(z1) or w(z2) and the halves of the field are added by one
// shuffle; else one lane evaluates both.  Called by full warps.  The step is
// one dependent chain from the position to the position; it holds no branch
// and no vote, so that the Gaussian factor and the scales are worked out
// beside the series.
template <bool PAIR>
__device__ __forceinline__ void walk_step(const StepRegs<PAIR>& st, int sub, bool active, double ba,
                                          double bb, IonState& q) {
  const double da = q.a - st.ma, db = q.b - st.mb;
  const double aa = fabs(da), ab = fabs(db);
  const double ua = aa * st.ga, ub = ab * st.gb;
  const double g = exp_neg(0.5 * fma(ua, ua, ub * ub));
  cplx f;
  if (PAIR) {
    f = weideman_scaled(aa * st.sa[0], ab * st.sb[0], sub ? -(st.c1 * g) : st.c1);
    f.re += __shfl_xor_sync(FULL_MASK, f.re, 1);
    f.im += __shfl_xor_sync(FULL_MASK, f.im, 1);
  } else {
    const double zr[2] = {aa * st.sa[0], aa * st.sa[1]}, zi[2] = {ab * st.sb[0], ab * st.sb[1]};
    cplx w[2];
    w_weideman_fast<2>(zr, zi, w);
    f = {st.c1 * fma(-g, w[1].re, w[0].re), st.c1 * fma(-g, w[1].im, w[0].im)};
  }
  double fa = da <= 0 ? -f.im : f.im, fb = db <= 0 ? -f.re : f.re;
  if (ua + ub < 1.0e-5) fa = fb = 0.0;  // MPBunch.cpp:1128
  walk_move(fa, fb, st.dt, active, ba, bb, q);
}

// The same for any bunch and any ion, one lane for both w(z), out of line: a
// round bunch, or an ion far from the bunch (|z| >= 30).
__device__ __noinline__ cplx walk_field_any(const WalkStep& st, double da, double db) {
  double fa, fb;
  if (st.mode == 2) {
    gaussian_round_field(da, db, 1.0 / st.ga, &fa, &fb);
    return {st.ci * fa, st.ci * fb};
  }
  const double aa = fabs(da), ab = fabs(db), ua = aa * st.ga, ub = ab * st.gb;
  const double zr[2] = {aa * st.sa[0], aa * st.sa[1]}, zi[2] = {ab * st.sb[0], ab * st.sb[1]};
  const double g = exp_neg(0.5 * fma(ua, ua, ub * ub));
  cplx w[2];
  w_quadrant1_wide2(zr, zi, w);
  const cplx f = {st.c1 * fma(-g, w[1].re, w[0].re), st.c1 * fma(-g, w[1].im, w[0].im)};
  return {da <= 0 ? -f.im : f.im, db <= 0 ? -f.re : f.re};
}

// The nw steps of a window for one ion born at step `born` of it (or before),
// its position at each step into the window's rows; flags: what walk_step_flags
// gives for the window's bunches.  Called by full warps.
template <bool PAIR, int ROW, int ACT>
__device__ __forceinline__ void walk_window(const WalkStep* s_st, int flags, int nw, int born,
                                            int sub, int slot, double (*s_x)[ROW],
                                            double (*s_y)[ROW], uint8_t (*s_act)[ACT], double bx,
                                            double by, IonState& q) {
  if (!__any_sync(FULL_MASK, q.alive && born < nw)) {
    if (sub == 0)
      for (int s = 0; s < nw; ++s) s_act[s][slot] = 0;
    return;
  }
  // ions start a call anywhere (a cloud kept from the last one, a birth)
  const bool inside = __all_sync(FULL_MASK, !q.alive || (fabs(q.a) <= bx && fabs(q.b) <= by));
  if (inside && (flags == kWinFlip || flags == kWinStay)) {
    if (flags == kWinFlip) {
      q.flip();
      double t = bx; bx = by; by = t;
      double(*r)[ROW] = s_x; s_x = s_y; s_y = r;
    }
    // PAIR, a lone chain: the next step's constants are loaded while this one's
    // runs (with one lane per ion other warps fill the wait)
    StepRegs<PAIR> cur = step_regs<PAIR>(s_st[0], sub), nxt;
#pragma unroll 1
    for (int s = 0; s < nw; ++s) {
      if (PAIR) nxt = step_regs<PAIR>(s_st[min(s + 1, nw - 1)], sub);
      else cur = step_regs<PAIR>(s_st[s], sub);
      const bool active = q.alive && s >= born;
      if (sub == 0) {  // the cloud bunch j sees: ions alive after the births of bunch j
        s_x[s][slot] = q.a;
        s_y[s][slot] = q.b;
        s_act[s][slot] = active ? 1 : 0;
      }
      walk_step<PAIR>(cur, sub, active, bx, by, q);
      if (PAIR) cur = nxt;
    }
    if (flags == kWinFlip) q.flip();
    return;
  }
#pragma unroll 1
  for (int s = 0; s < nw; ++s) {
    const bool active = q.alive && s >= born;
    if (sub == 0) {
      s_x[s][slot] = q.a;
      s_y[s][slot] = q.b;
      s_act[s][slot] = active ? 1 : 0;
    }
    const WalkStep& st = s_st[s];
    const bool sw = st.mode == 1;
    const double da = (sw ? q.b : q.a) - st.ma, db = (sw ? q.a : q.b) - st.mb;
    cplx f = walk_field_any(st, da, db);
    if (fabs(da) * st.ga + fabs(db) * st.gb < 1.0e-5) f = {0.0, 0.0};  // MPBunch.cpp:1128
    walk_move(sw ? f.im : f.re, sw ? f.re : f.im, st.dt, active, bx, by, q);
  }
}

// One CTA block = IONS trajectories (two lanes each) or, when the clouds hold
// enough ions to fill the GPU with one lane each (T > kWalkWide), 2 IONS
// trajectories: index t < n0 is ion t of the cloud the previous call left, t
// >= n0 the ion born as number (t - n0) % NM at bunch (t - n0) / NM.
// blockIdx.y = species.  The step loop has no block barrier: each ion's
// position at each step goes to a shared-memory window of kWin steps, and
// after each window the CTA sums it per step in a fixed order into the
// per-step partials.  A launch walks the bunch steps [ja, jb): trajectories
// that started before ja resume from the state the previous segment stored,
// so the walk can run as consecutive segments (the turn graph kicks the
// bunches of one segment while the next segment walks).
// A train of few ions is bound by the chain of one ion (0.38 us a step alone,
// of which the FP64 pipe issues 270 cycles), a large cloud by the FP64 pipe:
// 227 FP64 operations per ion and step with one lane, 2 x 136 with two, 4 x
// 165 in the form with four lanes per ion that this replaced.  200,000 ions
// through 1000 bunches: 19.7 -> 3.5 ms per interaction point; the 900-bunch
// train from empty clouds: 848 -> 521 us (prep to compaction).  The two forms and
// the slow path in one kernel of 128 registers spill 200 to 280 bytes: one
// instruction in thirty.
template <int IONS>
__global__ void __launch_bounds__(2 * IONS, 256 / IONS) k_ion_walk(ChainParams cp, IonWalk w,
                                                                 const CloudDev* __restrict__ clouds,
                                                                 const CloudState* __restrict__ cst,
                                                                 int ja, int jb) {
  constexpr int NT = 2 * IONS;
  constexpr int kGroups = NT / kWin;  // groups of ions summed per step
  constexpr int kRow = NT + 8;        // row stride: the rows of one half-warp in distinct banks
  __shared__ double s_x[kWin][kRow], s_y[kWin][kRow];
  __shared__ uint8_t s_act[kWin][NT];
  __shared__ double s_grp[kWin][kGroups][5];
  __shared__ WalkStep s_st[kWin];
  __shared__ int s_flags;
  const int p = blockIdx.y, G = gridDim.x, c = blockIdx.x;
  const int M = cp.n_bunches, NM = cp.macro_per_ip;
  const int n0 = cst[p].n;
  const int64_t T = (int64_t)n0 + (int64_t)M * NM;
  const bool wide = T > kWalkWide;
  const int per = wide ? NT : IONS;  // trajectories per block
  const int nblk = (int)((T + per - 1) / per);
  if (c >= nblk) return;
  const int tid = threadIdx.x, slot = wide ? tid : tid >> 1, sub = wide ? 0 : tid & 1;
  const CloudDev cd = clouds[p];
  const double bx = w.bound[0], by = w.bound[1];
  const double* births = w.births + 2 * (size_t)p * M * NM;
  const double* spec = w.spec + 2 * (size_t)p * M;
  double* part = w.part + (size_t)p * M * G * 5;
  double* traj = w.traj + (size_t)p * 6 * w.tcap;
  uint8_t* alive_out = w.alive + (size_t)p * w.tcap;
  bool first = true;
  for (int blk = c; blk < nblk; blk += G, first = false) {
    const int64_t t = (int64_t)blk * per + slot;
    const int64_t tb = (int64_t)blk * per;
    const int jfirst = tb < n0 ? 0 : (int)((tb - n0) / NM);
    const int js = max(jfirst, ja);
    if (first)
      for (int e = tid; e < 5 * (min(js, jb) - ja); e += NT)
        part[((size_t)(ja + e / 5) * G + c) * 5 + e % 5] = 0.0;
    IonState q = {0, 0, 0, 0, 0, 0, t < T};
    int j0 = 0;
    if (q.alive) {
      const int start = t < n0 ? 0 : (int)((t - n0) / NM);
      if (t >= n0) j0 = start;
      if (start < ja) {  // walked by an earlier segment
        q.a = traj[t];
        q.b = traj[w.tcap + t];
        q.va = traj[2 * w.tcap + t];
        q.vb = traj[3 * w.tcap + t];
        q.alive = alive_out[t] != 0;
      } else if (t < n0) {
        q.a = cd.x[0][t];
        q.b = cd.y[0][t];
        q.va = cd.vx[0][t];
        q.vb = cd.vy[0][t];
      } else {
        const int64_t b = t - n0;
        q.a = births[2 * b];
        q.b = births[2 * b + 1];
      }
    }
    for (int jw = js; jw < jb; jw += kWin) {
      const int nw = min(kWin, jb - jw);
      // the window's bunch constants in shared memory (global loads would sit
      // on the latency chain of every step)
      int flags = 0;
      if (tid < nw) {
        const int j = jw + tid;
        const WalkStep st = walk_step_of(w.prep[j], w.bunch + 3 * j, spec[2 * j + 1]);
        flags = walk_step_flags(st, bx, by);
        s_st[tid] = st;
      }
      if (tid < 32) {
        flags = __reduce_or_sync(FULL_MASK, flags);
        if (tid == 0) s_flags = flags;
      }
      __syncthreads();
      if (wide) walk_window<false>(s_st, s_flags, nw, j0 - jw, 0, slot, s_x, s_y, s_act, bx, by, q);
      else walk_window<true>(s_st, s_flags, nw, j0 - jw, sub, slot, s_x, s_y, s_act, bx, by, q);
      __syncthreads();
      {  // per step and group of ions: (count, sum x, sum y, sum x^2, sum y^2)
        const int s = tid / kGroups, g = tid % kGroups;
        if (s < nw) {
          double a[5] = {0, 0, 0, 0, 0};
          for (int i = g; i < per; i += kGroups) {
            if (!s_act[s][i]) continue;
            const double xi = s_x[s][i], yi = s_y[s][i];
            a[0] += 1.0;
            a[1] += xi;
            a[2] += yi;
            a[3] += xi * xi;
            a[4] += yi * yi;
          }
#pragma unroll
          for (int e = 0; e < 5; ++e) s_grp[s][g][e] = a[e];
        }
      }
      __syncthreads();
      for (int e = tid; e < 5 * nw; e += NT) {
        const int s = e / 5;
        double a = 0.0;
#pragma unroll
        for (int g = 0; g < kGroups; ++g) a += s_grp[s][g][e % 5];
        double* dst = part + ((size_t)(jw + s) * G + c) * 5 + e % 5;
        if (first) *dst = a;
        else *dst += a;
      }
    }
    if (t < T && sub == 0) {
      traj[t] = q.a;
      traj[w.tcap + t] = q.b;
      traj[2 * w.tcap + t] = q.va;
      traj[3 * w.tcap + t] = q.vb;
      traj[4 * w.tcap + t] = q.ka;
      traj[5 * w.tcap + t] = q.kb;
      alive_out[t] = q.alive ? 1 : 0;
    }
    __syncthreads();  // shared windows reused by the next block of this CTA
  }
}

// Records of the bunch steps [ja, jb), one warp per step and species: the
// partial sums of the walk's CTAs (each lane every 32nd CTA, then a butterfly:
// a fixed order) -> cloud centroid and rms -> the record the electron kick
// reads.  The one-ion quirk keeps the previous centroid, so the last CTA to
// finish carries the centroid through the steps that hold one ion and, across
// launches, in w.carry (initialised from the cloud state at ja = 0); at jb = M
// the last rms is kept there too, for the cloud state.
// As one CTA for all steps it took 223 us for a segment of 250 steps over 592
// walk CTAs (23 MB of partials through one SM).
__global__ void __launch_bounds__(kRecThreads) k_ion_records(ChainParams cp, IonWalk w,
                                                           const CloudState* __restrict__ cst,
                                                           CloudRec* rec, FieldPrep* rec_prep,
                                                           int* status, int G, int ions,
                                                           int ja, int jb) {
  __shared__ double s_ax[kRecChunk], s_ay[kRecChunk];
  __shared__ uint8_t s_one[kRecChunk];
  __shared__ double s_carry[2];
  __shared__ bool s_last;
  const int p = blockIdx.y, P = cp.n_species, tid = threadIdx.x, lane = tid & 31;
  const int M = cp.n_bunches, NM = cp.macro_per_ip;
  const CloudState st0 = cst[p];
  const int64_t T = (int64_t)st0.n + (int64_t)M * NM;
  const int per = T > kWalkWide ? 2 * ions : ions;
  const int nblk = (int)((T + per - 1) / per);
  const int nwork = nblk < G ? nblk : G;
  const double* spec = w.spec + 2 * (size_t)p * M;
  double* carry = w.carry + 4 * (size_t)p;
  const int j = ja + (int)blockIdx.x * (kRecThreads / 32) + (tid >> 5);
  if (j < jb) {
    const double* part = w.part + ((size_t)p * M + j) * G * 5;
    double s[5] = {0, 0, 0, 0, 0};
    for (int cc = lane; cc < nwork; cc += 32)
#pragma unroll
      for (int q = 0; q < 5; ++q) s[q] += part[5 * cc + q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < 5; ++q) s[q] += __shfl_xor_sync(FULL_MASK, s[q], o);
    if (lane == 0) {
      const int n = (int)s[0];
      double ax = 0, ay = 0, rx, ry;
      if (n == 1) {  // one ion: rms = |x| and the centroid stays (LIP.cpp:1125-1129)
        rx = fabs(s[1]);
        ry = fabs(s[2]);
      } else {
        const double inv_n = 1.0 / n;
        ax = s[1] * inv_n;
        ay = s[2] * inv_n;
        rx = sqrt(fmax(s[3] * inv_n - ax * ax, 0.0));
        ry = sqrt(fmax(s[4] * inv_n - ay * ay, 0.0));
      }
      if (n > cp.max_ions) atomicOr(status, kStatusIonOverflow);  // LIP.cpp:1043-1048
      CloudRec r;
      r.coeff = 2.0 * (spec[2 * j] * n) * kElecClassicRadius / cp.r_gamma;
      r.rms_x = rx;
      r.rms_y = ry;
      r.aver_x = ax;
      r.aver_y = ay;
      r.count = n;
      rec[(size_t)j * P + p] = r;
      // the field constants of this Gaussian, once for all the kicks that read it
      rec_prep[(size_t)j * P + p] = field_prep(rx, ry);
      if (j == M - 1) {
        carry[2] = rx;
        carry[3] = ry;
      }
    }
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&w.done[2 * p], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (tid == 0) {
    w.done[2 * p] = 0;
    s_carry[0] = ja == 0 ? st0.aver_x : carry[0];
    s_carry[1] = ja == 0 ? st0.aver_y : carry[1];
  }
  for (int j0 = ja; j0 < jb; j0 += kRecChunk) {
    const int nj = min(kRecChunk, jb - j0);
    bool one = false;
    __syncthreads();
    for (int jj = tid; jj < nj; jj += kRecThreads) {
      const CloudRec* r = rec + (size_t)(j0 + jj) * P + p;
      s_one[jj] = __ldcg(&r->count) == 1.0;
      s_ax[jj] = __ldcg(&r->aver_x);
      s_ay[jj] = __ldcg(&r->aver_y);
      one = one || s_one[jj];
    }
    if (!__syncthreads_or(one)) {  // no one-ion step: nothing to carry in
      if (tid == 0) {
        s_carry[0] = s_ax[nj - 1];
        s_carry[1] = s_ay[nj - 1];
      }
      continue;
    }
    if (tid == 0) {
      double cx = s_carry[0], cy = s_carry[1];
      for (int jj = 0; jj < nj; ++jj) {
        if (s_one[jj]) {
          s_ax[jj] = cx;
          s_ay[jj] = cy;
        } else {
          cx = s_ax[jj];
          cy = s_ay[jj];
        }
      }
      s_carry[0] = cx;
      s_carry[1] = cy;
    }
    __syncthreads();
    for (int jj = tid; jj < nj; jj += kRecThreads) {
      if (!s_one[jj]) continue;
      CloudRec* r = rec + (size_t)(j0 + jj) * P + p;
      r->aver_x = s_ax[jj];
      r->aver_y = s_ay[jj];
    }
  }
  if (tid == 0) {
    carry[0] = s_carry[0];
    carry[1] = s_carry[1];
  }
}

// After the last walk segment and the last records: the surviving ions in
// trajectory order (birth order, as the reference's erase keeps it) into
// cloud buffer 0, and the cloud state.  One CTA per kCompactThreads
// trajectories and species: it counts the survivors before its own by reading
// their flags (16 at a time) and keeps its own in order; the CTA that finishes
// last writes the state, when no other reads it any more.
// As one CTA it took 100 us for 20,000 ions, one round of barriers per 1024.
__global__ void __launch_bounds__(kCompactThreads) k_ion_compact(ChainParams cp, IonWalk w,
                                                              CloudDev* clouds, CloudState* cst,
                                                              int* status) {
  __shared__ int s_wsum[kCompactThreads / 32];
  __shared__ int s_before;
  const int p = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int M = cp.n_bunches, NM = cp.macro_per_ip;
  const CloudState st0 = cst[p];
  const int64_t T = (int64_t)st0.n + (int64_t)M * NM;
  const int64_t t0 = (int64_t)blockIdx.x * kCompactThreads;
  const CloudDev cd = clouds[p];
  if (t0 < T) {
    const double* traj = w.traj + (size_t)p * 6 * w.tcap;
    const uint8_t* al = w.alive + (size_t)p * w.tcap;
    if (tid == 0) s_before = 0;
    __syncthreads();
    int before = 0;  // flags are 0 or 1: a word's set bits are its survivors
    for (int64_t i = tid; i < t0 / 16; i += kCompactThreads) {
      const uint4 v = reinterpret_cast<const uint4*>(al)[i];
      before += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
    }
    before = __reduce_add_sync(FULL_MASK, before);
    if (lane == 0 && before) atomicAdd(&s_before, before);
    const int64_t t = t0 + tid;
    const bool keep = t < T && al[t];
    const unsigned bal = __ballot_sync(FULL_MASK, keep);
    if (lane == 0) s_wsum[warp] = __popc(bal);
    __syncthreads();
    int pre = s_before, tot = s_before;
    for (int u = 0; u < kCompactThreads / 32; ++u) {
      pre += u < warp ? s_wsum[u] : 0;
      tot += s_wsum[u];
    }
    pre += __popc(bal & ((1u << lane) - 1u));
    if (keep && pre < cd.cap) {
      cd.x[0][pre] = traj[t];
      cd.y[0][pre] = traj[w.tcap + t];
      cd.vx[0][pre] = traj[2 * w.tcap + t];
      cd.vy[0][pre] = traj[3 * w.tcap + t];
      cd.fx[pre] = traj[4 * w.tcap + t];
      cd.fy[pre] = traj[5 * w.tcap + t];
    }
    if (tid == 0 && t0 + kCompactThreads >= T) w.carry[4 * (size_t)cp.n_species + p] = tot;
  }
  __syncthreads();
  if (tid != 0) return;
  __threadfence();
  if (atomicAdd(&w.done[2 * p + 1], 1u) != gridDim.x - 1) return;
  __threadfence();
  w.done[2 * p + 1] = 0;
  const double* spec = w.spec + 2 * (size_t)p * M;
  const double* carry = w.carry + 4 * (size_t)p;
  const int total = (int)__ldcg(&w.carry[4 * (size_t)cp.n_species + p]);
  CloudState st;
  st.n = total < cd.cap ? total : cd.cap;
  if (total > cd.cap) atomicOr(status, kStatusIonOverflow);
  st.cur = 0;
  st.aver_x = carry[0];
  st.aver_y = carry[1];
  st.rms_x = carry[2];
  st.rms_y = carry[3];
  st.macro_charge = spec[2 * (M - 1)];
  cst[p] = st;
}

static ChainSection chain_section(const Handle& h, int k) {
  ChainSection cs;
  const cg_section& s = h.sections[k];
  cs.pressure = s.pressure;
  cs.temperature = s.temperature;
  cs.length = s.length;
  cs.aperture_x = s.aperture_x;
  cs.aperture_y = s.aperture_y;
  return cs;
}

cudaError_t launch_ion_prep(Handle& h, int k) {
  constexpr int kWarps = kPrepThreads / 32;
  k_ion_prep<<<(h.M * h.P + kWarps - 1) / kWarps, kPrepThreads, 0, h.stream>>>(
      h.chain, chain_section(h, k), h.d.bunch, h.d.mom, h.d.iw, h.d.status, h.d.turn, k);
  return cudaGetLastError();
}

// Shared memory a walk CTA of each shape asks for beyond its static arrays
// when its SM is reserved: together with the static arrays and the 1 KB the
// driver keeps per CTA, the whole 228 KB of the SM, so that no kick or map
// CTA is scheduled beside the walk (their warps would take issue slots and
// FP64 pipe cycles from the walk's latency-bound chain).  Set per device by
// prepare_ion_walk; index 0..2 = 16, 32, 64 ions per CTA.
static int g_walk_reserve_dyn[3] = {0, 0, 0};

template <int IONS>
static cudaError_t prepare_walk_shape(int slot) {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, k_ion_walk<IONS>);
  if (e != cudaSuccess) return e;
  const int dyn = 227 * 1024 - (int)a.sharedSizeBytes;
  e = cudaFuncSetAttribute(k_ion_walk<IONS>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn);
  if (e == cudaSuccess) g_walk_reserve_dyn[slot] = dyn;
  return e;
}

cudaError_t prepare_ion_walk() {
  cudaError_t e = prepare_walk_shape<16>(0);
  if (e == cudaSuccess) e = prepare_walk_shape<32>(1);
  if (e == cudaSuccess) e = prepare_walk_shape<64>(2);
  return e;
}

cudaError_t launch_ion_walk(Handle& h, int k, int ja, int jb, cudaStream_t s) {
  const int ions = std::max(16, h.walk_ions);  // 8 runs as 16: one warp
  const dim3 grid(ion_walk_grid(h.d.iw.tcap, ions), h.P);
  const CloudDev* cl = h.d.clouds + (size_t)k * h.P;
  const CloudState* cs = h.d.cloud_state + (size_t)k * h.P;
  const int slot = ions == 16 ? 0 : ions == 32 ? 1 : 2;
  const size_t dyn = h.walk_reserve ? (size_t)g_walk_reserve_dyn[slot] : 0;
  if (ions == 16) k_ion_walk<16><<<grid, 32, dyn, s>>>(h.chain, h.d.iw, cl, cs, ja, jb);
  else if (ions == 32) k_ion_walk<32><<<grid, 64, dyn, s>>>(h.chain, h.d.iw, cl, cs, ja, jb);
  else k_ion_walk<64><<<grid, 128, dyn, s>>>(h.chain, h.d.iw, cl, cs, ja, jb);
  return cudaGetLastError();
}

cudaError_t launch_ion_records(Handle& h, int k, int ja, int jb, cudaStream_t s) {
  constexpr int kWarps = kRecThreads / 32;
  const int ions = std::max(16, h.walk_ions);
  const dim3 grid((jb - ja + kWarps - 1) / kWarps, h.P);
  if (jb <= ja) return cudaSuccess;
  k_ion_records<<<grid, kRecThreads, 0, s>>>(h.chain, h.d.iw, h.d.cloud_state + (size_t)k * h.P,
                                             h.d.rec + (size_t)k * h.M * h.P,
                                             h.d.rec_prep + (size_t)k * h.M * h.P, h.d.status,
                                             ion_walk_grid(h.d.iw.tcap, ions), ions, ja, jb);
  return cudaGetLastError();
}

cudaError_t launch_ion_compact(Handle& h, int k, cudaStream_t s) {
  const dim3 grid((unsigned)((h.d.iw.tcap + kCompactThreads - 1) / kCompactThreads), h.P);
  k_ion_compact<<<grid, kCompactThreads, 0, s>>>(h.chain, h.d.iw, h.d.clouds + (size_t)k * h.P,
                                                 h.d.cloud_state + (size_t)k * h.P, h.d.status);
  return cudaGetLastError();
}

cudaError_t launch_ion_chain(Handle& h, int k) {
  cudaError_t e = launch_ion_prep(h, k);
  if (e == cudaSuccess) e = launch_ion_walk(h, k, 0, h.M, h.stream);
  if (e == cudaSuccess) e = launch_ion_records(h, k, 0, h.M, h.stream);
  if (e == cudaSuccess) e = launch_ion_compact(h, k, h.stream);
  return e;
}

cudaError_t upload_weideman_table_ion() {
  cudaError_t e = cudaMemcpyToSymbol(c_weideman, &h_weideman, sizeof(WeidemanTable));
  return e != cudaSuccess ? e : prepare_ion_walk();
}

// Latency floor of the walk: one warp advances 16 ions through a dependent
// chain of bunch passages with exactly the walk's step (walk_step) and none of
// its window stores, barriers and sums.  With coefficient 1e-13 the ion
// oscillates in the core of the Gaussian (period of ~300 passages), where the
// walk spends its time (Weideman region of w(z)).
__global__ void k_field_chain(double* out, int n) {
  const double bunch[3] = {0.0, 0.0, 1.0};
  const int sub = threadIdx.x & 1;
  const WalkStep st = walk_step_of(field_prep(1.4e-5, 6.3e-6), bunch, 1.0e-13);
  const StepRegs<true> r = step_regs<true>(st, sub);
  IonState q = {3.0e-6, 2.0e-6, 0.0, 0.0, 0.0, 0.0, true};
  for (int i = 0; i < n; ++i) walk_step<true>(r, sub, true, 1.0, 1.0, q);
  if (threadIdx.x == 0) out[0] = q.a + q.b;
}

cudaError_t measure_field_chain_latency(double* us_per_step) {
  double* out = nullptr;
  cudaError_t e = cudaMalloc(&out, sizeof(double));
  if (e != cudaSuccess) return e;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const int n = 4096;
  k_field_chain<<<1, 32>>>(out, 64);  // warm-up
  cudaEventRecord(e0);
  k_field_chain<<<1, 32>>>(out, n);
  cudaEventRecord(e1);
  e = cudaEventSynchronize(e1);
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  if (e != cudaSuccess) return e;
  *us_per_step = 1e3 * (double)ms / n;
  return cudaGetLastError();
}

int ion_walk_grid(int64_t tcap, int ions) {
  const int64_t blocks = (tcap + ions - 1) / ions;
  return (int)std::max<int64_t>(1, std::min<int64_t>(blocks, 148 * 4));
}

}  // namespace cg
