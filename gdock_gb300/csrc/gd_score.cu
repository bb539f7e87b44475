// The plain FP64 scoring kernel (the correctness form) and the per-call
// scoring set-up shared with the FP32 form (gd_score_warp.cu): the
// parameter block of a complex and the dispatch by precision.
//
// Reference arithmetic (gdock): transform src/structure.rs:80-131 and
// src/chromosome.rs:79-83; energies src/fitness.rs:57-302; per-pose
// combination src/chromosome.rs:110-127.
//
// k_score_f64: one pose per thread-block cluster of 1 to 16 CTAs.
//   1. The ligand's atoms are moved in FP64 with the reference's operation
//      order (coordinates bit-identical to gdock's) into shared memory, each
//      CTA of the cluster a share, the others copied from its shared memory.
//   2. Work units of one 32-atom ligand slot x a run of receptor atoms are
//      taken by the cluster's warps from one counter.  A unit finds its pairs
//      within reach in FP32 (bounding spheres of the slot and of the receptor
//      segments, then each pair's distance, all with the FP32 guard band
//      added, so that only pairs whose every term is exactly zero are dropped)
//      and lists them in shared memory; every 32 listed pairs are evaluated to
//      FP64 accuracy, one per lane: near pairs (within 12 A) every term, far
//      ones Coulomb only.  Distances and reciprocals are formed in integers,
//      which issue beside the slow FP64 pipe.  Decisions are exact: the squared
//      distance's high word settles them, and pairs next to a cutoff are
//      decided on d2 in the reference's operation order against the exact
//      thresholds.
//   3. Every term is added as a 128-bit fixed-point integer.  Integer sums are
//      exact, so the energies do not depend on which lane, warp or CTA took
//      which pair, nor on the launch's other poses.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "gd_device.cuh"

namespace gd {
namespace {

namespace cg = cooperative_groups;

constexpr int kNT = 256;              // threads per CTA of k_score_f64
constexpr int kNW = kNT / 32;
constexpr int kLigBits = 10;
constexpr int kLigCap = 1 << kLigBits;  // ligand atoms held in shared memory at once (longer ligands: in turns)
// Ligands up to this many atoms have their burial counts in shared memory from
// first to last; longer ones a turn at a time, in a variant of its own: the turn's
// end in the common one cost its pairs 2.5 % (registers), and the counts of longer
// ligands in shared memory cost a resident CTA.  300 poses on 2,538 atoms, all
// counts / a turn's: ligands of 3,000 atoms 2.16 / 2.38 ms, 4,200 2.87 / 3.18, 6,000
// 4.37 / 3.87, 20,000 11.3 / 9.6.
constexpr int kLigCounts = 4096;
constexpr int kRows = 4;              // rows searched per step
constexpr int kRowBuf = 32 + kRows;   // rows waiting per warp: fewer than a step and 32 more
constexpr int kQueue = 32 * (kRows + 1);  // listed pairs per warp and kind: 31 left over + 32 of each row
constexpr int kRowsMin = 8, kRowsMax = 128;  // receptor atoms of a unit (a power of two)
constexpr int kMaxCluster = 16;
constexpr unsigned kFixCoarse = 1u << 21;  // 1/8 A^2 as a fixed-point d2's high word
constexpr int kTinyHi = 0x2b000000;   // high word of 2^-335: below it r^6 may underflow

struct F64Smem {
  size_t x, y, z, q, fx, fy, fz, lt, sph, rcnt, lcnt, queue, row, red, nf, frame, misc, total;
};

__host__ __device__ inline F64Smem f64_smem(int nr, int nl, bool turns) {
  F64Smem L;
  size_t o = 0;
  const size_t cap = nl < kLigCap ? (static_cast<size_t>(nl) + 31) / 32 * 32 : kLigCap;
  auto take = [&](size_t b) {
    const size_t at = o;
    o += (b + 15) / 16 * 16;
    return at;
  };
  L.x = take(8 * cap);
  L.y = take(8 * cap);
  L.z = take(8 * cap);
  L.q = take(8 * cap);
  L.fx = take(4 * cap);
  L.fy = take(4 * cap);
  L.fz = take(4 * cap);
  L.lt = take(cap);
  L.sph = take(sizeof(float4) * (cap / 32));
  L.rcnt = take(2 * (static_cast<size_t>(nr) + 1));  // 16-bit burial counts, two a word
  L.lcnt = take(2 * ((turns ? cap : static_cast<size_t>(nl)) + 1));
  L.queue = take(2 * sizeof(uint32_t) * kQueue * kNW);
  L.row = take(sizeof(float4) * kRowBuf * kNW);
  L.red = take(3 * sizeof(__int128) * kNW);
  L.nf = take(3 * sizeof(double) * kNW);
  L.frame = take(sizeof(gd_pose_frame));
  L.misc = take(32);  // next unit, satisfied restraints, AIR energy
  L.total = o;
  return L;
}

// 1/d by one third-order step x (1 + e + e^2), e = 1 - d x (the Householder
// series of the reciprocal), on the hardware's approximation x, whose
// relative error is at most 2^-23: the remaining error e^3 lies below the
// FP64 rounding.  Three FP64 multiply-adds; FP64 issues at 1/64 of the FP32
// rate on this part, and a correctly rounded division costs about ten.
__device__ __forceinline__ double rcp64(double d) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
  double e = __fma_rn(-d, x, 1.0);
  e = __fma_rn(e, e, e);
  return __fma_rn(x, e, x);
}

// 1/d in integers, for normal d from 2^-1022 to 2^1021: with the significand
// M / 2^53 and the hardware's FP32 approximation Y / 2^23 of its reciprocal, the
// residual E = 2^76 - M Y is exact modulo 2^64 (it is below 2^55), and the
// reciprocal is Y (1 + e + e^2 + ...) with e = E / 2^76 below 2^-21, formed to
// 2^-57 and rounded once (0.51 units in the last place).  Some 33 integer
// instructions beside the FP64 pipe, in place of three on it.
__device__ __forceinline__ double rcp_int(double d) {
  const unsigned lo = static_cast<unsigned>(__double2loint(d)), hi = static_cast<unsigned>(__double2hiint(d));
  const unsigned mh = (hi & 0xfffffu) | 0x100000u;
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(__funnelshift_l(lo, mh, 3) + 0x3e800000u)));
  const unsigned Y = min(__float_as_uint(y) - 0x3f000000u, 0xffffffu);
  const long long E = -static_cast<long long>(static_cast<unsigned long long>(lo) * Y + (static_cast<unsigned long long>(mh * Y) << 32));
  const int eh = static_cast<int>(E >> 31);
  const unsigned el = static_cast<unsigned>(E >> 7) & 0xffffffu;
  const long long t = static_cast<long long>(eh) * static_cast<int>(Y) + __umulhi(Y << 8, el);
  const int s = eh >> 8;
  const unsigned q = __umulhi(static_cast<unsigned>(s * s), Y << 8) >> 11;
  const unsigned long long V = (static_cast<unsigned long long>(Y) << 39) + (t >> 6) + q;
  return __longlong_as_double(static_cast<long long>(((V + 512) >> 10) + (static_cast<unsigned long long>(2044 - (hi >> 20)) << 52)));
}
// ... and for any other d (infinite, undefined, next to the range's ends)
__device__ __noinline__ double rcp_rare(double d) { return rcp64(d); }

// min(count, 10) is all that is read: a count that has reached 10 is left
// alone, which also keeps the 16 bits from overflowing (at most 10 + one
// concurrent add of each of the CTA's threads).
__device__ __forceinline__ void bury(uint32_t *cnt, int i) {
  const int sh = (i & 1) * 16;
  if (((*reinterpret_cast<volatile uint32_t *>(cnt + (i >> 1)) >> sh) & 0xffffu) < 10u) atomicAdd(cnt + (i >> 1), 1u << sh);
}

// A pair's d2 in the reference's arithmetic and its decisions: bit 0 vdW, 1
// burial, 2 Coulomb, 3: r^6 underflows and R6 is zero, where the reference's
// ratio is 0 / 0.  Kept out of line: a handful of pairs in a million come
// here, and inlined as predicated instructions they took a third of the FP64
// pipe.
struct ExactPair {
  double d2;
  int flags;
};
__device__ __noinline__ ExactPair exact_pair(const ScoreParams &p, const gd_pose_frame &f, int pose, int ri, int j) {
  const D4 r = p.rec_pos64[ri];
  double X, Y, Z;
  ligand_atom(p, f, pose, j, X, Y, Z);
  const double d2 = exact_d2(r.x, r.y, r.z, X, Y, Z);
  const Thresholds &t = p.thr;
  ExactPair e{d2, (d2 > 0.0 && d2 < t.vdw_lt) | (d2 < t.desolv_lt) << 1 | (d2 > t.elec_gt && d2 < t.elec_lt) << 2};
  if ((e.flags & 1) && d2 * d2 * d2 == 0.0 && signbit(p.tab64[p.rec_meta[ri].x + p.lig_type[j]].inv2)) e.flags |= 8;
  return e;
}

// A double's high word next to that of the squared cutoff t (a relative 2^-20
// to either side: more than the few ulps between a fused d2 and the
// reference's).
__device__ __forceinline__ bool near_hi(int hi, double t) {
  return static_cast<unsigned>(hi - (__double2hiint(t) - 1)) <= 2u;
}
// FIX: d2 from integer coordinates of 2^-51 A.  Doubles from 2 A on lie on that
// grid; a smaller coordinate moves by 2^-52 A at most, of the order of what the
// transform's own roundings leave.  The differences and the three squares are
// exact and d2 is truncated below 2^-56 A^2, half a unit in a double's last place
// from 1/8 A^2 on; closer pairs (a few in a million) are formed in FP64 in the
// reference's order.  It takes about 45 integer instructions a pair, which issue
// beside the FP64 pipe, in place of 6 FP64 ones.
template <bool FIX, bool SERIAL, bool CLAMP, bool TURNS>
struct PairEval {
  const ScoreParams &p;
  const gd_pose_frame &f;
  int pose;
  const void *x, *y, *z;  // FIX: integers, else doubles
  const double *q;
  const uint8_t *lt;
  uint32_t *rcnt, *lcnt;
  int base;  // ligand atom of the shared arrays' first entry

  // one listed pair per lane (on): w = receptor atom, ligand entry
  template <bool NEAR>
  __device__ __forceinline__ void eval(bool on, uint32_t w, ExactSum<> &vdw, ExactSum<> &elec) const {
    if (!on) return;
    const int ri = static_cast<int>(w >> kLigBits), k = static_cast<int>(w & (kLigCap - 1));
    double rq, d2;
    bool pv, pd, pe, rare;
    if (FIX) {
      const longlong2 *rp = reinterpret_cast<const longlong2 *>(p.rec_fix + ri);
      const longlong2 rxy = __ldg(rp), rzq = __ldg(rp + 1);
      rq = __longlong_as_double(rzq.y);
      const long long d[3] = {rxy.x - static_cast<const long long *>(x)[k], rxy.y - static_cast<const long long *>(y)[k],
                              rzq.x - static_cast<const long long *>(z)[k]};
      const unsigned long long D = fix_d2(d);  // 2^-56 A^2
      const unsigned hw = static_cast<unsigned>(D >> 32);
      // to a double, rounded: the leading bit at 63 - n (n = 0 from 128 A^2 on)
      const int n = NEAR ? __clz(hw) : 0;
      const unsigned long long m = D << n;
      d2 = __longlong_as_double(static_cast<long long>((m >> 11) + ((m >> 10) & 1)) +
                                (static_cast<long long>(1029 - n) << 52));
      pe = hw < (225u << 24);
      rare = near_fix(hw, 225u);
      if (NEAR) {
        pv = hw < (144u << 24);
        pd = hw < (64u << 24);
        pe = pe && hw >= (1u << 24);
        rare = rare | near_fix(hw, 144u) | near_fix(hw, 64u) | near_fix(hw, 1u) | (hw < kFixCoarse);
      }
    } else {
      const double2 *rp = reinterpret_cast<const double2 *>(p.rec_pos64 + ri);
      const double2 rxy = __ldg(rp), rzq = __ldg(rp + 1);
      rq = rzq.y;
      const double dx = rxy.x - static_cast<const double *>(x)[k], dy = rxy.y - static_cast<const double *>(y)[k],
                   dz = rzq.x - static_cast<const double *>(z)[k];
      d2 = __fma_rn(dz, dz, __fma_rn(dy, dy, dx * dx));
      const int hi = __double2hiint(d2);
      pe = hi < __double2hiint(p.thr.elec_lt);
      rare = near_hi(hi, p.thr.elec_lt);
      if (NEAR) {
        pv = hi < __double2hiint(p.thr.vdw_lt);
        pd = hi < __double2hiint(p.thr.desolv_lt);
        pe = pe && hi > __double2hiint(p.thr.elec_gt);
        // a zero, a tiny or an undefined d2 (NaN: hi < 0) takes the exact tests too
        rare = rare | near_hi(hi, p.thr.vdw_lt) | near_hi(hi, p.thr.desolv_lt) | near_hi(hi, p.thr.elec_gt) | (hi < kTinyHi);
      }
    }
    if (rare) {
      const ExactPair e = exact_pair(p, f, pose, ri, base + k);
      d2 = e.d2;
      pv = e.flags & 1;
      pd = e.flags & 2;
      pe = e.flags & 4;
      if (e.flags & 8) vdw.nf = NAN;
    }
    if (NEAR) {
      const int2 m = __ldg(p.rec_meta + ri);
      if (SERIAL) pv = pv && m.y != __ldg(p.lig_serial + base + k);
      if (pd) {
        bury(rcnt, ri);
        bury(lcnt, TURNS ? k : base + k);
      }
      if (pv) {
        // softcore_lj_potential (src/fitness.rs:57-70) as 4 eps (x^2 - x) with
        // x = 1 / (r^6 2/R6 + 1), half the reference's ratio
        const double2 tp = __ldg(reinterpret_cast<const double2 *>(p.tab64) + m.x + lt[k]);
        const double w = __fma_rn(d2 * d2 * d2, tp.x, 1.0);
        const double u = static_cast<unsigned>(__double2hiint(w)) < 0x7fc00000u ? rcp_int(w) : rcp_rare(w);
        double v = tp.y * __fma_rn(u, u, -u);
        if (CLAMP) v = v < -50.0 ? -50.0 : (v > 500.0 ? 500.0 : v);
        vdw.add_term(v, p.fx_vdw);
      }
    }
    // elec_energy term (src/fitness.rs:296) without its constant, which
    // multiplies the pose's sum
    if (pe) elec.add_term(rq * q[k] * rcp_int(d2), p.fx_elec);
  }
};

// What bounds it: the FP64 pipe (two lanes' operations per clock and SM; 55 %
// busy) and instruction issue (63 %), at the 24 warps an SM that the registers
// allow.  The form that evaluated every pair spent about 35 FP64 operations on
// each pair, though only 13 % of the pairs of a scan have a term; a listed pair
// cost 18 (near) or 11 (far), 6 fewer with d2 from integers, and with the
// reciprocals in integers too it is 7 or 2.  The FP32 search takes some 25
// instructions a row of 32 pairs: rows wait in shared memory as position and
// list entry, and two of five of its pairs are listed.  On receptors of 2,538
// and ligands of 1,280 atoms: 2,048 poses 348 -> 28.7 -> 18.7 -> 12.4 ms (every
// pair; listed pairs; d2 from integers; reciprocals, short sums, row buffer), 150
// poses 29.0 -> 2.38 -> 1.72 -> 1.40 ms; one pose of 411 x 649 atoms 1,746 -> 89
// -> 53 us a call.
template <bool FIX, bool SERIAL, bool CLAMP, bool TURNS>
__global__ void __launch_bounds__(kNT, 3) k_score_f64(const ScoreParams p, const int unit_rows) {
  if (p.skip && *p.skip) return;
  extern __shared__ __align__(128) unsigned char smem[];
  const F64Smem L = f64_smem(p.nr, p.nl, TURNS);
  double *s_x = reinterpret_cast<double *>(smem + L.x), *s_y = reinterpret_cast<double *>(smem + L.y),
         *s_z = reinterpret_cast<double *>(smem + L.z), *s_q = reinterpret_cast<double *>(smem + L.q);
  float *s_fx = reinterpret_cast<float *>(smem + L.fx), *s_fy = reinterpret_cast<float *>(smem + L.fy),
        *s_fz = reinterpret_cast<float *>(smem + L.fz);
  uint8_t *s_lt = smem + L.lt;
  float4 *s_sph = reinterpret_cast<float4 *>(smem + L.sph);
  uint32_t *s_rcnt = reinterpret_cast<uint32_t *>(smem + L.rcnt), *s_lcnt = reinterpret_cast<uint32_t *>(smem + L.lcnt);
  gd_pose_frame *s_frame = reinterpret_cast<gd_pose_frame *>(smem + L.frame);
  __int128 *s_red = reinterpret_cast<__int128 *>(smem + L.red);
  double *s_nf = reinterpret_cast<double *>(smem + L.nf);
  int *s_next = reinterpret_cast<int *>(smem + L.misc), *s_sat = s_next + 1;
  double *s_air = reinterpret_cast<double *>(smem + L.misc + 8);

  cg::cluster_group cluster = cg::this_cluster();
  const int nc = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int pose = static_cast<int>(blockIdx.x) / nc;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  uint32_t *q_near = reinterpret_cast<uint32_t *>(smem + L.queue) + warp * 2 * kQueue, *q_far = q_near + kQueue;
  float4 *s_row = reinterpret_cast<float4 *>(smem + L.row) + warp * kRowBuf;

  if (!p.models && tid < 16)
    reinterpret_cast<double *>(s_frame)[tid] = reinterpret_cast<const double *>(p.frames + pose)[tid];
  for (int i = tid; i < (p.nr + 1) / 2; i += kNT) s_rcnt[i] = 0;
  for (int i = tid; i < ((TURNS ? min(p.nl, kLigCap) : p.nl) + 1) / 2; i += kNT) s_lcnt[i] = 0;
  if (TURNS && lane == 0) {
    s_red[warp * 3 + 2] = 0;
    s_nf[warp * 3 + 2] = 0.0;
  }
  if (tid == 0) *s_next = 0;
  __syncthreads();
  const gd_pose_frame &f = *s_frame;

  // FP32 reach of the elec and vdW cutoffs with their guard bands.  The tests
  // below are written so that an undefined comparison (coordinates beyond
  // FP32) and an infinite band keep the pair for the FP64 decision.
  const float lim_e = 225.0f + p.guard_e, lim_v = 144.0f + p.guard_v;
  const float reach = sqrtf(225.01f + 2.0f * p.guard_e) + 0.01f;
  const int ngrp = (p.nr + unit_rows - 1) / unit_rows;
  ExactSum<> vdw, elec;
  int first = 0;  // unit counter at the start of this turn

  const int turns = (p.nl + kLigCap - 1) / kLigCap, turn = turns ? ((p.nl + turns - 1) / turns + 31) / 32 * 32 : 0;
  for (int l0 = 0; l0 < p.nl; l0 += turn) {
    const int nl = min(turn, p.nl - l0), nslot = (nl + 31) / 32, nunit = nslot * ngrp;
    // the CTA's share of the slots: one warp per slot, one atom per lane
    for (int s = rank + nc * warp; s < nslot; s += nc * kNW) {
      const int k = s * 32 + lane, j = l0 + k;
      const bool on = k < nl;
      bool held = on;  // in the sphere
      float fx = 0.0f, fy = 0.0f, fz = 0.0f;
      if (on) {
        double X, Y, Z;
        ligand_atom(p, f, pose, j, X, Y, Z);
        fx = static_cast<float>(X - p.ox);
        fy = static_cast<float>(Y - p.oy);
        fz = static_cast<float>(Z - p.oz);
        if (FIX) {
          // The receptor lies within kFixMax, so an atom with a coordinate beyond
          // kFixHold, or one that is not a number, has no pair with a term: images
          // at infinity keep it out of the search.  A property of the atom alone:
          // the launch's other poses, and what their displacements are said to
          // be, change nothing.
          held = fabs(X) < kFixHold && fabs(Y) < kFixHold && fabs(Z) < kFixHold;
          if (!held) {
            X = Y = Z = 0.0;
            fx = fy = fz = INFINITY;
          }
          constexpr double kOne = 1LL << kFixBits;
          s_x[k] = __longlong_as_double(__double2ll_rn(X * kOne));
          s_y[k] = __longlong_as_double(__double2ll_rn(Y * kOne));
          s_z[k] = __longlong_as_double(__double2ll_rn(Z * kOne));
        } else {
          s_x[k] = X;
          s_y[k] = Y;
          s_z[k] = Z;
        }
        s_fx[k] = fx;
        s_fy[k] = fy;
        s_fz[k] = fz;
      }
      // a sphere around the slot: the precomputed smallest one moved with the
      // pose, else the bounding box's centre and farthest atom
      float lo[3] = {held ? fx : 3.0e38f, held ? fy : 3.0e38f, held ? fz : 3.0e38f},
            hi[3] = {held ? fx : -3.0e38f, held ? fy : -3.0e38f, held ? fz : -3.0e38f};
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          lo[a] = fminf(lo[a], __shfl_xor_sync(kFull, lo[a], o));
          hi[a] = fmaxf(hi[a], __shfl_xor_sync(kFull, hi[a], o));
        }
      const float cx = 0.5f * (lo[0] + hi[0]), cy = 0.5f * (lo[1] + hi[1]), cz = 0.5f * (lo[2] + hi[2]);
      float rr = held ? sqrtf((fx - cx) * (fx - cx) + (fy - cy) * (fy - cy) + (fz - cz) * (fz - cz)) : 0.0f;
      const bool odd = __any_sync(kFull, !(rr < 3.0e38f));  // not finite: a sphere that keeps everything
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) rr = fmaxf(rr, __shfl_xor_sync(kFull, rr, o));
      if (lane == 0) {
        float4 sp = make_float4(cx, cy, cz, odd ? INFINITY : rr * 1.0001f + 0.01f);
        if (!p.models && !odd) {
          const D4 v = p.lig_slot_sph[(l0 >> 5) + s];
          double x, y, z;
          relative_atom(p, f, v, x, y, z);
          const float r = static_cast<float>(v.w) * 1.0001f + 0.01f;
          if (r < sp.w) sp = make_float4(static_cast<float>(x), static_cast<float>(y), static_cast<float>(z), r);
        }
        s_sph[s] = sp;
      }
    }
    for (int k = tid; k < nl; k += kNT) {
      int t = p.lig_type[l0 + k];
      if (!GD_DCHECK(p.err, t >= 0 && t < p.nt, 22)) t = 0;
      s_lt[k] = static_cast<uint8_t>(t);
      s_q[k] = p.lig_q[l0 + k];
    }
    if (nc > 1) {
      // the other CTAs' slots, out of their shared memory
      cluster.sync();
      for (int s = warp; s < nslot; s += kNW) {
        const int o = s % nc;
        if (o == rank) continue;
        const int k = s * 32 + lane;
        if (k < nl) {
          s_x[k] = *cluster.map_shared_rank(s_x + k, o);
          s_y[k] = *cluster.map_shared_rank(s_y + k, o);
          s_z[k] = *cluster.map_shared_rank(s_z + k, o);
          s_fx[k] = *cluster.map_shared_rank(s_fx + k, o);
          s_fy[k] = *cluster.map_shared_rank(s_fy + k, o);
          s_fz[k] = *cluster.map_shared_rank(s_fz + k, o);
        }
        if (lane == 0) s_sph[s] = *cluster.map_shared_rank(s_sph + s, o);
      }
    }
    __syncthreads();

    const PairEval<FIX, SERIAL, CLAMP, TURNS> ev{p, f, pose, s_x, s_y, s_z, s_q, s_lt, s_rcnt, s_lcnt, l0};
    int *next = nc > 1 ? cluster.map_shared_rank(s_next, 0) : s_next;
    int nn = 0, nf = 0;  // listed near and far pairs of this warp
    for (;;) {
      int u = 0;
      if (lane == 0) u = atomicAdd(next, 1);
      u = __shfl_sync(kFull, u, 0) - first;
      if (u >= nunit) break;
      const int slot = u / ngrp, r0 = u % ngrp * unit_rows, r1 = min(p.nr, r0 + unit_rows);
      const int k = slot * 32 + lane;
      const bool on = k < nl;
      const float lx = on ? s_fx[k] : 0.0f, ly = on ? s_fy[k] : 0.0f, lz = on ? s_fz[k] : 0.0f;
      const float4 sp = s_sph[slot];
      const float lim_s = sp.w + reach, lim_s2 = lim_s * lim_s;
      int nrow = 0;  // rows waiting
      // kRows waiting rows (n of them real) against the lane's atom: their
      // loads, distances and votes overlap
      auto step = [&](int at, int n) {
        float4 r[kRows];
        float d2[kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) r[i] = s_row[at + i];
#pragma unroll
        for (int i = 0; i < kRows; ++i) d2[i] = d2f(r[i], lx, ly, lz);
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
          const bool reached = on && i < n && !(d2[i] > lim_e), close = reached && !(d2[i] > lim_v);
          const unsigned Mn = __ballot_sync(kFull, close), Mf = __ballot_sync(kFull, reached && !close);
          const int to = (close ? nn : kQueue + nf) + __popc((close ? Mn : Mf) & lt_mask);
          if (reached) q_near[to] = __float_as_uint(r[i].w) | static_cast<uint32_t>(k);
          nn += __popc(Mn);
          nf += __popc(Mf);
        }
        if (nn >= 32 || nf >= 32) {
          __syncwarp();
          for (; nn >= 32; nn -= 32) ev.template eval<true>(true, q_near[nn - 32 + lane], vdw, elec);
          for (; nf >= 32; nf -= 32) ev.template eval<false>(true, q_far[nf - 32 + lane], vdw, elec);
          __syncwarp();
        }
      };
#pragma unroll 1
      for (int a0 = r0 & ~31;; a0 += 32) {
        const bool last = a0 >= r1;
        if (!last) {
          {
            const float4 sg = __ldg(&p.rec_seg[a0 / kRecSeg]);
            const float dx = sg.x - sp.x, dy = sg.y - sp.y, dz = sg.z - sp.z;
            const float lim = sg.w + sp.w + reach + 0.1f + 1e-3f * (sg.w + sp.w);
            if (dx * dx + dy * dy + dz * dz > lim * lim) {
              a0 |= 32;  // the segment's second half too
              continue;
            }
          }
          // rows: receptor atoms within reach of the slot's sphere
          bool keep = a0 + lane >= r0 && a0 + lane < r1;
          float4 r = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (keep) {
            r = __ldg(&p.rec_pos32[a0 + lane]);
            const float dx = r.x - sp.x, dy = r.y - sp.y, dz = r.z - sp.z;
            keep = !(dx * dx + dy * dy + dz * dz > lim_s2);
          }
          const unsigned rows = __ballot_sync(kFull, keep);
          if (keep) {
            r.w = __uint_as_float(static_cast<uint32_t>(a0 + lane) << kLigBits);
            s_row[nrow + __popc(rows & lt_mask)] = r;
          }
          nrow += __popc(rows);
          __syncwarp();
        }
        int at = 0;
        for (; at + kRows <= nrow; at += kRows) step(at, kRows);
        if (last) {
          if (at < nrow) step(at, nrow - at);
          break;
        }
        if (at > 0) {  // fewer than a step are left
          nrow -= at;
          __syncwarp();
          if (lane < nrow) s_row[lane] = s_row[at + lane];
        }
      }
      __syncwarp();
    }
    // the rest of both lists, together when they fit one round (the near
    // evaluation decides every term itself)
    __syncwarp();
    if (nn + nf <= 32) {
      ev.template eval<true>(lane < nn + nf, lane < nn ? q_near[lane] : q_far[lane - nn], vdw, elec);
    } else {
      ev.template eval<true>(lane < nn, q_near[lane], vdw, elec);
      ev.template eval<false>(lane < nf, q_far[lane], vdw, elec);
    }
    __syncwarp();
    // every warp of the cluster drew one unit number past the last
    first += nunit + nc * kNW;
    if (l0 + turn < p.nl) {
      if (nc > 1) cluster.sync();  // nobody reads this turn's ligand atoms any more
      else __syncthreads();
      if constexpr (TURNS) {
        // a turn's atoms have met every receptor atom: their counts are complete
        ExactSum<> part;
        for (int i = rank * kNT + tid; i < nl; i += nc * kNT) {
          unsigned c = 0;
          for (int r = 0; r < nc; ++r) c += (cluster.map_shared_rank(s_lcnt, r)[i >> 1] >> ((i & 1) * 16)) & 0xffffu;
          part.add(p.lig_desolv[static_cast<size_t>(l0 + i) * 11 + min(c, 10u)], p.fx_desolv);
        }
        part.warp_total();
        if (lane == 0) {
          s_red[warp * 3 + 2] += part.v;
          s_nf[warp * 3 + 2] += part.nf;
        }
        if (nc > 1) cluster.sync();
        else __syncthreads();
        for (int i = tid; i < (nl + 1) / 2; i += kNT) s_lcnt[i] = 0;
      }
    }
  }

  // AIR: one restraint per lane, summed in restraint order (bit-identical)
  if (rank == 0 && warp == 0) {
    double air;
    int sat;
    warp_air(p, f, pose, lane, air, sat);
    if (lane == 0) {
      *s_air = air;
      *s_sat = sat;
    }
  }
  if (nc > 1) cluster.sync();
  else __syncthreads();
  // desolvation from the cluster's summed burial counts, a share per CTA
  ExactSum<> desolv;
  const int l_left = TURNS && turn ? (p.nl - 1) / turn * turn : 0;  // first ligand atom not summed yet
  for (int side = 0; side < 2; ++side) {
    const int n = side ? p.nl - l_left : p.nr;
    const double *tab = side ? p.lig_desolv + static_cast<size_t>(l_left) * 11 : p.rec_desolv;
    uint32_t *cnt = side ? s_lcnt : s_rcnt;
    for (int i = rank * kNT + tid; i < n; i += nc * kNT) {
      unsigned c = 0;
      for (int r = 0; r < nc; ++r) {
        const uint32_t *o = nc > 1 ? cluster.map_shared_rank(cnt, r) : cnt;
        c += (o[i >> 1] >> ((i & 1) * 16)) & 0xffffu;
      }
      desolv.add(tab[static_cast<size_t>(i) * 11 + min(c, 10u)], p.fx_desolv);
    }
  }
  vdw.warp_total();
  elec.warp_total();
  desolv.warp_total();
  if (lane == 0) {
    if (TURNS) {
      desolv.v += s_red[warp * 3 + 2];
      desolv.nf += s_nf[warp * 3 + 2];
    }
    s_red[warp * 3] = vdw.v;
    s_red[warp * 3 + 1] = elec.v;
    s_red[warp * 3 + 2] = desolv.v;
    s_nf[warp * 3] = vdw.nf;
    s_nf[warp * 3 + 1] = elec.nf;
    s_nf[warp * 3 + 2] = desolv.nf;
  }
  if (nc > 1) cluster.sync();
  else __syncthreads();
  if (rank == 0 && tid < 32) {
    ExactSum<> t[3];
    for (int w = lane; w < nc * kNW; w += 32)
      for (int c = 0; c < 3; ++c) {
        const int at = (w % kNW) * 3 + c;
        t[c].v += nc > 1 ? *cluster.map_shared_rank(s_red + at, w / kNW) : s_red[at];
        t[c].nf += nc > 1 ? *cluster.map_shared_rank(s_nf + at, w / kNW) : s_nf[at];
      }
    for (int c = 0; c < 3; ++c) t[c].warp_total();
    if (lane == 0)
      write_pose(p, pose, t[0].value(p.fx_vdw), 332.0636 * t[1].value(p.fx_elec), t[2].value(p.fx_desolv), *s_air, *s_sat);
  }
  if (nc > 1) cluster.sync();  // the shared memory read above stays until here
}

// ------------------------------------------------------------ dispatch ----

template <typename Kern>
cudaError_t launch_f64(Kern kern, const ScoreParams &p, bool turns, int sm_count, cudaStream_t stream) {
  const size_t smem = f64_smem(p.nr, p.nl, turns).total;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  // CTAs per pose: the more the fewer poses there are, as far as the pose's
  // rows (receptor atom x ligand slot) go round.  Poses differ widely in work,
  // so splitting them pays beyond the point where they fill the SMs, the less
  // so the more CTAs a cluster must find places for at once.  Measured (the
  // call), us at 1 / 2 / 4 / 8 / 16 CTAs: 2,538 x 1,280 atoms, 40 poses 2714 /
  // 1461 / 776 / 495 / 529, 300 poses 3515 / 2811 / 2414 / 2382 / 3169, 1,200
  // poses 8544 / 7867 / 7850 / 8810 / 12327; 411 x 649 atoms, 2,400 poses 2165 /
  // 2244 / 2648 / 3216 / 5165, 9,600 poses 7189 / 7996 / 9966 / 12375 / 20207;
  // 253 x 170 atoms, one pose 69 / 53 / 42 / 40 / 39.
  const long long rows = static_cast<long long>(std::max(1, (std::min(p.nl, kLigCap) + 31) / 32)) * std::max(1, p.nr);
  constexpr int kPerSm[] = {64, 32, 16, 4};  // CTAs per SM up to which poses are split in 2, 4, 8, 16
  int nc = 1;
  for (int k = 0; k < 4 && nc < kMaxCluster; ++k)
    if (static_cast<long long>(p.n_poses) * (2 << k) <= static_cast<long long>(kPerSm[k]) * sm_count &&
        rows > 16 * kNW * (2 << k))
      nc = 2 << k;
  // rows per unit: 32 units or more for every warp, so that the last ones
  // leave few warps waiting (8 to 128 units a warp made no difference)
  int unit_rows = kRowsMin;
  while (unit_rows < kRowsMax && rows >= 2LL * unit_rows * 32 * kNW * nc) unit_rows *= 2;
  if (nc > 8) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(kNT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  for (;; nc /= 2) {
    at.val.clusterDim.x = static_cast<unsigned>(nc);
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3(static_cast<unsigned>(p.n_poses) * nc);
    if (nc == 1) break;
    // a cluster this large may not fit beside the shared memory it needs
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) == cudaSuccess && fit > 0) break;
    (void)cudaGetLastError();
  }
  if (nc == 1) cfg.numAttrs = 0;
  return cudaLaunchKernelEx(&cfg, kern, p, unit_rows);
}

}  // namespace

ScoreParams make_params(gd_complex *cx, const gd_pose_frame *d_frames, const double *d_models, int n,
                        gd_pose_energy *d_out, double max_disp) {
  ScoreParams p{};
  p.rec_pos32 = cx->rec_pos32;
  p.rec_pos64 = cx->rec_pos64;
  p.rec_fix = cx->rec_fix;
  p.fix = cx->fix64;
  p.rec_meta = cx->rec_meta;
  p.rec_desolv = cx->rec_desolv;
  p.nr = cx->nr;
  p.lig_perm = cx->lig_perm;
  p.lig_slot_sph = cx->lig_slot_sph;
  p.lig_rel = cx->lig_rel;
  p.lig_fix = cx->lig_fix;
  p.fix32 = cx->fix32;
  std::copy(cx->ofix, cx->ofix + 3, p.ofix);
  p.rec_seg = cx->rec_seg;
  p.nseg = cx->nseg;
  p.lig_x = cx->lig_x;
  p.lig_y = cx->lig_y;
  p.lig_z = cx->lig_z;
  p.lig_q = cx->lig_q;
  p.lig_type = cx->lig_type;
  p.lig_serial = cx->lig_serial;
  p.lig_desolv = cx->lig_desolv;
  p.nl = cx->nl;
  p.cx = cx->cx;
  p.cy = cx->cy;
  p.cz = cx->cz;
  p.ox = cx->ox;
  p.oy = cx->oy;
  p.oz = cx->oz;
  p.tab32 = cx->tab32;
  p.tab64 = cx->tab64;
  p.fx_vdw = cx->fx_vdw;
  p.fx_elec = cx->fx_elec;
  p.fx_desolv = cx->fx_desolv;
  p.nt = cx->nt;
  p.need_clamp = cx->need_clamp;
  p.restr_rec = cx->restr_rec;
  p.restr_lig = cx->restr_lig;
  p.K = cx->K;
  p.wv = cx->w.vdw;
  p.we = cx->w.elec;
  p.wd = cx->w.desolv;
  p.wa = cx->w.air;
  p.thr = make_thresholds(5.0);
  guard_widths(cx, max_disp, &p.guard_v, &p.guard_e, &p.guard_d);
  p.frames = d_frames;
  p.models = d_models;
  p.n_poses = n;
  p.out = d_out;
  p.err = cx->ctx->d_err;
  return p;
}

gd_status launch_score(gd_complex *cx, const gd_pose_frame *d_frames, const double *d_models, int n,
                       gd_precision prec, gd_pose_energy *d_out, cudaStream_t stream, double max_disp,
                       const int *skip) {
  gd_context *ctx = cx->ctx;
  if (n <= 0) return GD_OK;
  ScoreParams p = make_params(cx, d_frames, d_models, n, d_out, max_disp);
  p.skip = skip;
  const bool serial = cx->serial_overlap, clamp = cx->need_clamp;
  if (prec == GD_PREC_F32)
    return launch_score_batch_f32(ctx, std::vector<ScoreParams>{p}, serial, clamp,
                                  ctx->tune_f32_slots ? ctx->tune_f32_slots : kDefaultF32Tune, stream);
  // Here the bands only keep FP32 from dropping a pair that has a term, and such
  // a pair's ligand atom lies within 15 A of the receptor's extent, wherever the
  // launch's poses are.  They are first order in the coordinates' FP32 rounding:
  // beyond 1 A^2 (receptor coordinates some 40,000 A from the origin, or not
  // finite) FP32 drops nothing and every pair is decided in FP64.
  guard_bands(cx->rec_extent + 17.0, &p.guard_v, &p.guard_e, &p.guard_d);
  if (!(p.guard_e <= 1.0f)) p.guard_e = p.guard_v = INFINITY;
  cudaError_t e;
  const int sm = ctx->sm_count;
  if (p.nl > kLigCounts) {
    // (one variant: the tests of the others change nothing where they are not needed)
    e = p.fix ? launch_f64(k_score_f64<true, true, true, true>, p, true, sm, stream)
              : launch_f64(k_score_f64<false, true, true, true>, p, true, sm, stream);
  } else if (p.fix) {
    if (serial) e = clamp ? launch_f64(k_score_f64<true, true, true, false>, p, false, sm, stream)
                          : launch_f64(k_score_f64<true, true, false, false>, p, false, sm, stream);
    else e = clamp ? launch_f64(k_score_f64<true, false, true, false>, p, false, sm, stream)
                   : launch_f64(k_score_f64<true, false, false, false>, p, false, sm, stream);
  } else {
    if (serial) e = clamp ? launch_f64(k_score_f64<false, true, true, false>, p, false, sm, stream)
                          : launch_f64(k_score_f64<false, true, false, false>, p, false, sm, stream);
    else e = clamp ? launch_f64(k_score_f64<false, false, true, false>, p, false, sm, stream)
                   : launch_f64(k_score_f64<false, false, false, false>, p, false, sm, stream);
  }
  if (e != cudaSuccess) {
    // the one size that the form does not take: the receptor's burial counts
    const size_t need = f64_smem(p.nr, p.nl, p.nl > kLigCounts).total;
    int most = 0;
    if (cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) == cudaSuccess &&
        need > static_cast<size_t>(most)) {
      const std::string what = "score kernel launch: a receptor of " + std::to_string(p.nr) + " atoms takes " +
                               std::to_string(need) + " bytes of shared memory a block, there are " + std::to_string(most);
      return cuda_fail(ctx, e, what.c_str());
    }
    return cuda_fail(ctx, e, "score kernel launch");
  }
  return GD_OK;
}

}  // namespace gd
