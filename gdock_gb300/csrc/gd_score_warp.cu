// Batched FP32 scoring: a persistent kernel in which every warp owns whole
// work items taken from a global queue, so that poses of many complexes of
// uneven sizes share one launch and no warp ever waits for another.  A work
// item is one pose, or (split mode, the default) one 128-atom ligand chunk of
// a pose, or for launches with few poses one receptor part of such a chunk
// (the receptor segments g with g mod R = part).
//
// Per work item a warp
//   1. copies the complex's descriptor and the pose frame to its shared memory;
//   2. for each chunk of 32*S ligand atoms: moves them in fixed point (nine
//      32-bit multiply-adds a coordinate, closer than FP64; out of its range in
//      FP64; src/structure.rs:80-131), keeps FP32
//      copies in shared memory (S slots of 32 atoms, one per lane; the ligand
//      is stored in spatially compact slot order) and a bounding sphere and
//      box per slot;
//   3. streams the receptor through its own two-stage shared-memory ring,
//      each stage filled by one bulk (TMA) copy of a 64-atom segment and
//      guarded by a per-warp mbarrier with a bounded wait; the receptor is
//      stored as spatially compact segments with bounding spheres, and only
//      the segments within reach of the chunk's slot spheres are copied and
//      tested (the slot spheres are precomputed and move rigidly with the
//      pose);
//   4. row test: each lane takes one (receptor atom, slot) row of an 8 x 4
//      round; a row whose atom lies beyond the 15 A reach of the slot's
//      sphere or box is dropped (every pair of it contributes exactly
//      nothing), one beyond the 12 A reach is a far row (Coulomb only); kept
//      rows go to per-slot lists in shared memory;
//   5. evaluates the kept rows four at a time (independent FP32 chains), the
//      last one or two of a slot two at a time: soft-core LJ, Coulomb, burial
//      counts and guard-band tests for near rows, Coulomb and its band for far
//      rows.  The kernel issues on 85 % of its cycles and no other unit is
//      near its limit, so instructions per row set its time: the slots' FP32
//      atoms lie in shared memory behind one loop (not one unrolled copy a
//      slot), and a list entry already holds the shared address of the row's
//      position and its row of the pair table.  That took 150 poses of
//      2,538 x 1,280 atoms from 419 to 376 us and 65,536 of them from 83.4
//      to 81.4 ms;
//   6. re-decides, once per segment, the pairs of flagged steps whose FP32 d2
//      lies within the guard band of a cutoff (1, 8, 12, 15 A): on integer
//      distances, and in the reference's FP64 order where those lie next to
//      the cutoff, so all decisions equal the FP64 ones;
//   7. reduces exactly: each segment's FP32 vdW and Coulomb partials become
//      2^-32 fixed-point integers summed per lane (integer sums do not depend
//      on their order, so neither do the energies on how segments, chunks and
//      receptor parts are grouped into work items), desolvation from the
//      exact burial counts in FP64 in a fixed order, AIR in restraint order
//      (bit-identical), and writes the six-field record
//      (src/chromosome.rs:110-127).  Split mode: the item that completes a
//      pose adds the items' partials.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "gd_device.cuh"

namespace gd {
namespace {

constexpr int kWarps = 4;      // warps per CTA (independent)
constexpr int kSeg = 64;       // receptor atoms per ring stage
constexpr int kWS = 2;         // ring stages per warp (a stage takes microseconds to process: two hide the copy)
constexpr int kBlk = 8;        // receptor atoms per row-test round (lane = slot * 8 + atom)
constexpr int kMaxS = 4;       // ligand slots per lane, at most (one row-test round covers 8 atoms x 4 slots)
constexpr int kList = kSeg + 8;  // row-list entries per slot: a segment's atoms + two paddings of 4 rows
constexpr int kFar = kWS * kSeg; // shared-memory index of the far-away dummy receptor atom
constexpr int kCntSmemMax = 4096;  // burial counters kept in shared memory up to this many receptor atoms
constexpr int kSegListMax = 512;   // receptor segments a chunk's culled list holds (more: every segment)
static_assert(kSeg == kRecSeg, "the ring stage is one receptor segment");

struct BatchParams {
  const ScoreParams *descs;       // one per complex
  const long long *item_start;    // prefix sums of work items, ncx + 1 entries
  int ncx;
  long long total;
  unsigned long long *queue;      // work counter, zero at launch
  uint8_t *gcounts;               // per-warp burial counters in global memory (when not in smem)
  int gcount_stride;              // bytes per warp in gcounts
  int smem_cnt;                   // bytes per warp of shared-memory counters (0: use gcounts)
  int max_nr;                     // largest receptor of the batch
  int *err;
  // split mode: a work item is one ligand chunk of a pose; the chunk that
  // finishes a pose last reduces its per-chunk partials
  int split;
  const long long *pose_start;    // first batch-wide pose index of each complex
  int max_chunks;                 // partial slots per pose (chunks x rparts)
  double2 *air;                   // [pose] restraint energy and satisfied restraints (rparts > 1)
  double *part;                   // [pose][chunk * rparts + part][vdw, elec (fixed point), ligand desolvation][32 lanes]
  unsigned *pcount;               // [pose][(max_nr + 1) / 2] receptor burial counts, two 16-bit counts a word
  int *pdone;                     // [pose] items finished
  int rparts;                     // receptor parts per chunk (split mode; 1: whole receptor)
  unsigned *lcount;               // [pose][max_nl] ligand burial counts (rparts > 1)
  int max_nl;
  // failure-detection test (GD_TUNE_FAULT): the warp that takes work item 0
  // issues no copy for its first ring stage, so its bounded wait runs out
  int drop_copy;
};

struct WarpSmem {
  size_t pos, meta, list, fixq, cmask, cstep, lig, lt, lcnt, bars, desc, frame, fixm, blob, box, rc, ssph, segl, cnt, total;
};

// atoms: rows per step of the kernel variant
__host__ __device__ inline WarpSmem warp_layout(int smem_cnt, int atoms) {
  WarpSmem L;
  size_t o = 0;
  auto al = [&](size_t a) { o = (o + a - 1) / a * a; };
  const size_t steps = kMaxS * (kList / atoms + 2);  // of a segment, at most
  L.pos = o;
  o += sizeof(float4) * (kWS * kSeg + 1);  // + the far dummy atom
  al(16);
  L.meta = o;
  o += sizeof(int2) * (kWS * kSeg + 1);
  al(16);
  L.list = o;   // kept rows per slot: shared address of the position << 12 | type row
  o += sizeof(uint32_t) * kMaxS * kList;
  al(16);
  L.fixq = o;   // flagged steps
  o += sizeof(uint16_t) * steps;
  al(16);
  L.cmask = o;  // per recorded near row of the segment: lanes with d2 < 64 (ballot)
  o += sizeof(unsigned) * kMaxS * kList;
  al(16);
  L.cstep = o;  // ... and per recorded step its place in the lists
  o += sizeof(uint16_t) * steps;
  al(16);
  L.lig = o;    // the chunk's ligand atoms (x, y, z, charge), their types and burial counts
  o += sizeof(float4) * kMaxS * 32;
  L.lt = o;
  o += sizeof(uint16_t) * kMaxS * 32;
  al(16);
  L.lcnt = o;
  o += sizeof(int) * kMaxS * 32;
  al(16);
  L.bars = o;
  o += 8 * kWS;
  al(16);
  L.desc = o;
  o += sizeof(ScoreParams);
  al(16);
  L.frame = o;
  o += sizeof(gd_pose_frame);
  L.fixm = o;  // the frame in fixed point: nine matrix entries, the translation
  o += 9 * sizeof(Limbs) + 3 * sizeof(long long);
  al(16);
  L.blob = o;
  o += sizeof(float4) * 8;
  L.box = o;
  o += sizeof(float4) * 2 * kMaxS;
  L.rc = o;
  o += sizeof(int) * kSeg;
  L.ssph = o;  // the chunk's slot spheres (culling test of the receptor segments)
  o += sizeof(float4) * kMaxS;
  L.segl = o;  // the chunk's receptor segments within reach
  o += sizeof(uint16_t) * kSegListMax;
  al(16);
  L.cnt = o;
  o += smem_cnt;
  al(128);
  L.total = o;
  return L;
}

__device__ __forceinline__ void issue_seg(long long q, int seg, const ScoreParams &p, float4 *s_pos, int2 *s_meta,
                                          uint64_t *s_bar) {
  const int st = static_cast<int>(q % kWS);
  constexpr uint32_t kBytes = kSeg * (sizeof(float4) + sizeof(int2));
  mbar_expect_tx(&s_bar[st], kBytes);
  bulk_g2s(&s_pos[st * kSeg], p.rec_pos32 + static_cast<size_t>(seg) * kSeg, kSeg * sizeof(float4), &s_bar[st]);
  bulk_g2s(&s_meta[st * kSeg], p.rec_meta + static_cast<size_t>(seg) * kSeg, kSeg * sizeof(int2), &s_bar[st]);
}

// acc += v when t < 0 (one predicated add)
__device__ __forceinline__ void add_if_lt0(float &acc, float t, float v) {
  asm("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %1, 0f00000000;\n\t@p add.f32 %0, %0, %2;\n\t}" : "+f"(acc)
      : "f"(t), "f"(v));
}
// acc = a * b + acc (one rounding) when t < 0
__device__ __forceinline__ void fma_if_lt0(float &acc, float t, float a, float b) {
  asm("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %1, 0f00000000;\n\t@p fma.rn.f32 %0, %2, %3, %0;\n\t}" : "+f"(acc)
      : "f"(t), "f"(a), "f"(b));
}
// acc = a * b + acc (one rounding) when |t| < lim
__device__ __forceinline__ void fma_if_abs_lt(float &acc, float t, float lim, float a, float b) {
  asm("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %1, %2;\n\t@p fma.rn.f32 %0, %3, %4, %0;\n\t}" : "+f"(acc)
      : "f"(fabsf(t)), "f"(lim), "f"(a), "f"(b));
}
// soft-core LJ in FP32 (src/fitness.rs:57-70): eps*(q^2 - 2q) with
// q = R6/(r^6 + R6/2), evaluated as 4 eps x (x - 1) = 4 eps (x^2 - x),
// x = q/2 = 1/(r^6 2/R6 + 1); at d2 = 0 it is exactly 0
template <bool CLAMP>
__device__ __forceinline__ float vdw_term(float d2, float2 tp) {
  const float r6 = d2 * d2 * d2;
  const float x = rcp_approx(__fmaf_rn(r6, tp.x, 1.0f));
  float v = __fmaf_rn(x, x, -x) * tp.y;
  if (CLAMP) v = v < -50.0f ? -50.0f : (v > 500.0f ? 500.0f : v);
  return v;
}

// One pair's FP32 terms.  The Coulomb sum accumulates q_r / d2 (scaled by
// the lane's ligand charge once per segment).  The vdW decision is d2 < 144
// alone: the reference's 0 < r excludes only coincident atoms, whose FP32 d2 is
// 0 (models) or within the rounding of the two images (poses, moved in fixed
// point: some 1e-11 A^2), where r^6 vanishes beside R6 and x^2 - x is exactly 0,
// so the sums are unchanged; the guard band of the vdW cutoff is the one at 144.
template <bool SERIAL, bool CLAMP>
__device__ __forceinline__ void pair32(float d2, float qr, const float2 tp, bool same, float gv, float ge, float gdd,
                                       float &av, float &ae, bool &amb) {
  const float tv = __fsub_rn(d2, 144.0f);  // d2 < 144  <=>  tv < 0
  if (SERIAL || CLAMP) {
    const float v = vdw_term<CLAMP>(d2, tp);
    if (SERIAL) av += (tv < 0.0f && !same) ? v : 0.0f;
    else add_if_lt0(av, tv, v);
  } else {
    // the well depth multiplies into the sum: one FMA (vdw_term without the
    // product's own rounding)
    const float x = rcp_approx(__fmaf_rn(d2 * d2 * d2, tp.x, 1.0f));
    fma_if_lt0(av, tv, __fmaf_rn(x, x, -x), tp.y);
  }
  const float te = __fsub_rn(d2, 113.0f);  // 1 < d2 < 225  <=>  |te| < 112
  fma_if_abs_lt(ae, te, 112.0f, qr, rcp_approx(d2));
  amb = amb | (fabsf(__fsub_rn(fabsf(te), 112.0f)) < ge) | (fabsf(tv) < gv) | (fabsf(__fsub_rn(d2, 64.0f)) < gdd);
}

__device__ __forceinline__ bool near_band(float d2, float gv, float ge, float gdd) {
  const float tv = __fsub_rn(d2, 144.0f), te = __fsub_rn(d2, 113.0f);
  return (fabsf(__fsub_rn(fabsf(te), 112.0f)) < ge) | (fabsf(tv) < gv) | (fabsf(__fsub_rn(d2, 64.0f)) < gdd);
}

__device__ __forceinline__ float3 atom32(const ScoreParams &p, const gd_pose_frame &f, int pose, int j) {
  double x, y, z;
  if (p.models) {
    ligand_atom(p, f, pose, j, x, y, z);
    x -= p.ox;
    y -= p.oy;
    z -= p.oz;
  } else {
    relative_atom(p, f, p.lig_rel[j], x, y, z);
  }
  return make_float3(static_cast<float>(x), static_cast<float>(y), static_cast<float>(z));
}

// Warp-wide minimum and maximum, one instruction each (volatile: every lane takes
// part, so the compiler must not sink them into a branch).
__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// Corrections of one pair's FP32 contributions after its exact re-decision.
struct FixOut {
  float dv, de;
  int dl;
};

// A pair's decisions in the reference's arithmetic: bit 0 vdW, 1 Coulomb, 2
// burial.  Out of line: a handful of pairs come here.
__device__ __noinline__ int exact_flags(const ScoreParams &p, const gd_pose_frame &f, int pose, int j, int ridx) {
  const D4 r64 = p.rec_pos64[ridx];
  double X, Y, Z;
  ligand_atom(p, f, pose, j, X, Y, Z);
  const double d2x = exact_d2(r64.x, r64.y, r64.z, X, Y, Z);
  return (d2x > 0.0 && d2x < p.thr.vdw_lt) | (d2x > p.thr.elec_gt && d2x < p.thr.elec_lt) << 1 | (d2x < p.thr.desolv_lt) << 2;
}

// Re-decision of one flagged pair (the lane's ligand atom j): recomputes the
// FP32 d2 and decisions bit-identically to pair32() and returns the corrections
// where the exact decision differs.  With the frame in fixed point (fm, ft) the
// integer d2 decides all but pairs within 6e-8 A^2 of a cutoff, which take the
// reference's FP64 order (some 45 FP64 operations, each 64 cycles apart): one
// pose of 2,538 x 1,280 atoms 88 -> 86 us, 65,536 poses 82.9 -> 82.6 ms.
template <bool SERIAL, bool CLAMP>
__device__ __forceinline__ FixOut fix_pair(const ScoreParams &p, const gd_pose_frame &f, int pose, int j, bool fix,
                                           const Limbs *fm, const long long *ft, float4 r, int ridx, int rtrow, int rser,
                                           float lx, float ly, float lz, float lq, int lt, int lser) {
  FixOut o{0.0f, 0.0f, 0};
  const float d2 = d2f(r, lx, ly, lz);
  const float te = __fsub_rn(d2, 113.0f);
  bool pv32 = __fsub_rn(d2, 144.0f) < 0.0f;
  if (SERIAL) pv32 = pv32 && (rser != lser);
  const bool pe32 = fabsf(te) < 112.0f;
  const bool pd32 = d2 < 64.0f;
  bool pv64 = false, pe64 = false, pd64 = false, decided = false;
  // (integers hold d2 below 256 A^2; pairs farther off come here where a pose of
  // the launch is so far away that the bands cover every distance)
  if (fix && d2 < 240.0f) {
    const int4 xy = __ldg(&p.lig_fix[2 * j]), z = __ldg(&p.lig_fix[2 * j + 1]);
    const longlong2 *rp = reinterpret_cast<const longlong2 *>(p.rec_fix + ridx);
    const longlong2 rxy = __ldg(rp);
    const long long rz = __ldg(reinterpret_cast<const long long *>(rp + 1));
    const long long d[3] = {rxy.x - p.ofix[0] - ft[0] - rotate(fm[0], fm[1], fm[2], xy, z),
                            rxy.y - p.ofix[1] - ft[1] - rotate(fm[3], fm[4], fm[5], xy, z),
                            rz - p.ofix[2] - ft[2] - rotate(fm[6], fm[7], fm[8], xy, z)};
    const unsigned hw = static_cast<unsigned>(fix_d2(d) >> 32);
    decided = !(near_fix(hw, 225u) | near_fix(hw, 144u) | near_fix(hw, 64u) | near_fix(hw, 1u) | (hw == 0u));
    pv64 = hw < (144u << 24);
    pd64 = hw < (64u << 24);
    pe64 = hw >= (1u << 24) && hw < (225u << 24);
  }
  if (!decided) {
    const int e = exact_flags(p, f, pose, j, ridx);
    pv64 = e & 1;
    pe64 = e & 2;
    pd64 = e & 4;
  }
  if (SERIAL) pv64 = pv64 && (rser != lser);
  if (pv64 != pv32) {
    const float v = vdw_term<CLAMP>(d2, __ldg(reinterpret_cast<const float2 *>(p.tab32) + rtrow + lt));
    o.dv = pv64 ? v : -v;
  }
  if (pe64 != pe32) {
    const float e = (r.w * rcp_approx(d2)) * lq;
    o.de = pe64 ? e : -e;
  }
  if (pd64 != pd32) o.dl = pd64 ? 1 : -1;
  return o;
}

// A segment's FP32 energy partial as a 2^-32 fixed-point integer.  Integer
// sums are exact, so the energies do not depend on how the segments are
// grouped into work items (whole poses, chunks, receptor parts) nor on the
// order the partials arrive in.  A segment's partial covers at most 256 pairs
// (64 receptor atoms x 4 lanes' slots) whose soft-core LJ terms are bounded
// by their well depths and Coulomb terms by 332 q q; a partial of 2^24
// kcal/mol or more (or not a number) is reported instead of wrapped.
__device__ __forceinline__ long long fx_energy(float x, int *err) {
  if (!(fabsf(x) < 16777216.0f)) {
    atomicCAS(err, 0, kDevRange);
    return 0;
  }
  return __float2ll_rn(x * 4294967296.0f);
}

__device__ __forceinline__ long long warp_sum_ll(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

__device__ __forceinline__ void bump_count(uint8_t *cnt, int i, int delta) {
  const int c = static_cast<int>(cnt[i]) + delta;
  cnt[i] = static_cast<uint8_t>(c > 255 ? 255 : (c < 0 ? 0 : c));
}

// SPLIT: 0 whole poses, 1 ligand chunks, 2 ligand chunks in receptor parts
// (bp.rparts; a separate instantiation keeps the single-part kernel's loops
// free of the part arithmetic)
template <int S, int kAtoms, int MINB, bool SERIAL, bool CLAMP, int SPLIT>
__global__ void __launch_bounds__(kWarps * 32, MINB) k_score_f32w(const BatchParams bp) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const WarpSmem L = warp_layout(bp.smem_cnt, kAtoms);
  unsigned char *base = smem + static_cast<size_t>(wib) * L.total;
  float4 *s_pos = reinterpret_cast<float4 *>(base + L.pos);
  int2 *s_meta = reinterpret_cast<int2 *>(base + L.meta);
  uint32_t *s_list = reinterpret_cast<uint32_t *>(base + L.list);
  uint16_t *s_fixq = reinterpret_cast<uint16_t *>(base + L.fixq);    // steps: list position | slot << 8 | rows << 12
  unsigned *s_cmask = reinterpret_cast<unsigned *>(base + L.cmask);
  uint16_t *s_cstep = reinterpret_cast<uint16_t *>(base + L.cstep);
  float4 *s_lig = reinterpret_cast<float4 *>(base + L.lig);
  uint16_t *s_lt = reinterpret_cast<uint16_t *>(base + L.lt);
  int *s_lcnt = reinterpret_cast<int *>(base + L.lcnt);
  uint64_t *s_bar = reinterpret_cast<uint64_t *>(base + L.bars);
  ScoreParams *s_desc = reinterpret_cast<ScoreParams *>(base + L.desc);
  gd_pose_frame *s_frame = reinterpret_cast<gd_pose_frame *>(base + L.frame);
  Limbs *s_fm = reinterpret_cast<Limbs *>(base + L.fixm);
  long long *s_ft = reinterpret_cast<long long *>(s_fm + 9);
  float4 *s_blob = reinterpret_cast<float4 *>(base + L.blob);
  float4 *s_box = reinterpret_cast<float4 *>(base + L.box);  // per slot: (centre, hx), (hy, hz, -, -)
  int *s_rc = reinterpret_cast<int *>(base + L.rc);  // receptor burial counts of the current segment
  float4 *s_ssph = reinterpret_cast<float4 *>(base + L.ssph);
  uint16_t *s_segl = reinterpret_cast<uint16_t *>(base + L.segl);
  // a list entry's parts (shared addresses fit 18 bits, type rows 12)
  const uint32_t pos_at = smem_u32(s_pos), far_row = (pos_at + kFar * 16) << 12;
  auto entry_atom = [&](uint32_t e) { return static_cast<int>(((e >> 12) - pos_at) >> 4); };
  static_assert(kMaxTypes * kMaxTypes <= 4096, "a type row in 12 bits");
  const int gwarp = static_cast<int>(blockIdx.x) * kWarps + wib;
  uint8_t *cnt = bp.smem_cnt ? reinterpret_cast<uint8_t *>(base + L.cnt)
                             : bp.gcounts + static_cast<size_t>(gwarp) * bp.gcount_stride;

  if (lane == 0) {
    for (int s = 0; s < kWS; ++s) mbar_init(&s_bar[s], 1);
    fence_mbar_init();
    s_pos[kFar] = make_float4(1.0e9f, 1.0e9f, 1.0e9f, 0.0f);  // far from real and idle ligand lanes
    s_meta[kFar] = make_int2(0, 0);
  }
  if (!SPLIT)
    for (int i = lane; i < bp.max_nr; i += 32) cnt[i] = 0;
  for (int i = lane; i < kSeg; i += 32) s_rc[i] = 0;
  __syncwarp();

  static_assert(S >= 1 && S <= kMaxS, "one row-test round covers at most four slots");
  constexpr int kChunk = 32 * S;
  const int my_s = lane >> 3, my_a = lane & 7;
  const unsigned my_group = 0xffu << (8 * my_s), lt_mask = (1u << lane) - 1u;
  long long q = 0;  // ring uses of this warp so far
  for (;;) {
    unsigned long long item = 0;
    if (lane == 0) item = atomicAdd(bp.queue, 1ull);
    item = __shfl_sync(kFull, item, 0);
    if (static_cast<long long>(item) >= bp.total) break;
    // complex of this item: last c with item_start[c] <= item
    int lo = 0, hi = bp.ncx - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (bp.item_start[mid] <= static_cast<long long>(item)) lo = mid;
      else hi = mid - 1;
    }
    const long long kk = static_cast<long long>(item) - bp.item_start[lo];
    __syncwarp();
    {
      const uint64_t *src = reinterpret_cast<const uint64_t *>(bp.descs + lo);
      uint64_t *dst = reinterpret_cast<uint64_t *>(s_desc);
      for (int w = lane; w < static_cast<int>(sizeof(ScoreParams) / 8); w += 32) dst[w] = src[w];
    }
    __syncwarp();
    const ScoreParams &p = *s_desc;
    if (p.skip && *p.skip) continue;  // this complex is finished (e.g. a converged GA job)
    // split mode: item = (pose, chunk, receptor part), at least one chunk per
    // pose (an empty ligand's single chunk holds no atom); otherwise item =
    // pose
    const int R = SPLIT == 2 ? bp.rparts : 1;
    const int nchunks = SPLIT ? max(1, (p.nl + kChunk - 1) / kChunk) : (p.nl + kChunk - 1) / kChunk;
    const int per_pose = nchunks * R;
    const int pose = static_cast<int>(SPLIT ? kk / per_pose : kk);
    const int rem = SPLIT ? static_cast<int>(kk % per_pose) : 0;
    const int ch0 = rem / R, rpart = rem % R;
    const int ch1 = SPLIT ? ch0 + 1 : nchunks;
    const int gp = SPLIT ? static_cast<int>(bp.pose_start[lo]) + pose : 0;  // poses of a launch fit an int
    if (!p.models && lane < 16)
      reinterpret_cast<double *>(s_frame)[lane] = reinterpret_cast<const double *>(p.frames + pose)[lane];
    __syncwarp();
    const gd_pose_frame &f = *s_frame;
    const int nseg = (p.nr + kSeg - 1) / kSeg;
    long long q_issued = q;  // ring uses issued so far (lane 0 issues; read on failure)
    const float gv = p.guard_v, ge = p.guard_e, gdd = p.guard_d;
    // a row (receptor atom, ligand slot) whose atom lies farther than this
    // from the slot's bounding sphere has every FP32 d2 beyond the elec
    // cutoff and its guard band: all its terms, counts and guard tests are 0
    const float reach = sqrtf(225.01f + 2.0f * ge) + 0.01f;
    // ... and one farther than this has every FP32 d2 beyond the vdW cutoff
    // and its band (so beyond the desolvation one too): Coulomb terms only
    const float reach_v = sqrtf(144.01f + 2.0f * gv) + 0.01f;
    const float reach2 = reach * reach, reach_v2 = reach_v * reach_v;
    const float2 *tab = reinterpret_cast<const float2 *>(p.tab32);
    long long vdw_i = 0, elec_i = 0;  // 2^-32 fixed point
    double desolv_t = 0.0;
    bool failed = false;

    for (int ch = ch0; ch < ch1 && !failed; ++ch) {
      // Receptor segments within reach of the chunk: each slot's precomputed
      // sphere moves rigidly with the pose (its centre transformed exactly),
      // and a segment whose sphere lies beyond the elec reach of every slot
      // sphere holds only rows the row test would drop.  Explicit model
      // coordinates (no rigid pose) keep every segment.
      const bool cull = p.models == nullptr && p.lig_slot_sph != nullptr && p.rec_seg != nullptr;
      if (cull && lane < S) {
        const int sl = ch * S + lane;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
        if (sl * 32 < p.nl) {
          const D4 sp = p.lig_slot_sph[sl];
          double x, y, z;
          relative_atom(p, f, sp, x, y, z);
          v = make_float4(static_cast<float>(x), static_cast<float>(y), static_cast<float>(z), static_cast<float>(sp.w));
        }
        s_ssph[lane] = v;
      }
      __syncwarp();
      // this item's segments: those of its receptor part (g mod R = part),
      // culled for a rigid pose
      const int nseg_part = (nseg - rpart + R - 1) / R;
      int nk = nseg_part;
      bool listed = false;
      if (cull) {
        nk = 0;
        for (int g0 = 0; g0 < nseg; g0 += 32) {
          const int g = g0 + lane;
          bool keep = false;
          if (g < nseg && g % R == rpart) {
            const float4 sg = __ldg(&p.rec_seg[g]);
#pragma unroll
            for (int s2 = 0; s2 < S; ++s2) {
              const float4 ss = s_ssph[s2];
              const float dx = sg.x - ss.x, dy = sg.y - ss.y, dz = sg.z - ss.z;
              const float lim = sg.w + ss.w + reach + 0.1f + 1e-3f * (sg.w + ss.w);
              keep = keep || (ss.w >= 0.0f && dx * dx + dy * dy + dz * dz < lim * lim);
            }
          }
          const unsigned m = __ballot_sync(kFull, keep);
          const int pos = nk + __popc(m & lt_mask);
          if (keep && pos < kSegListMax) s_segl[pos] = static_cast<uint16_t>(g);
          nk += __popc(m);
        }
        listed = nk <= kSegListMax;
        if (!listed) nk = nseg_part;  // too many to list: every segment of the part
        __syncwarp();
      }
      auto seg_at = [&](int k) { return listed ? static_cast<int>(s_segl[k]) : rpart + k * R; };
      long long fv = 0, fe = 0;  // this item's vdW and Coulomb sums, 2^-32 fixed point
#pragma unroll
      for (int s = 0; s < S; ++s) s_lcnt[s * 32 + lane] = 0;
      // an item without a segment in reach (the usual one of a pose apart from
      // the receptor, and of a receptor part) ends here
      if (nk > 0) {
        if (lane == 0)
          for (int k = 0; k < nk && k < kWS; ++k)
            if (!(bp.drop_copy && item == 0 && ch == ch0 && k == 0))
              issue_seg(q + k, seg_at(k), p, s_pos, s_meta, s_bar);
        q_issued = q + min(nk, kWS);
        // the frame in fixed point, an entry a lane.  With receptor parts every
        // part's item moves its ligand atoms, and in FP64 that kept its pipe 30 %
        // busy and the warps waiting: 150 poses of 2,538 x 1,280 atoms 347 ->
        // 330 us, of 1,074 x 741 176 -> 160, of 411 x 649 116 -> 103
        bool fix = p.fix32 && !p.models;
        if (fix) {
          bool ok = true;
          if (lane < 9) {
            const double a = lane == 0 ? f.ca : lane == 1 ? f.m01 : lane == 2 ? f.m02 : lane == 3 ? f.sa : lane == 4 ? f.m11
                             : lane == 5 ? f.m12 : lane == 6 ? -f.sb : f.cb;
            const double b = lane == 0 || lane == 3 ? f.cb : lane == 7 ? f.sg : lane == 8 ? f.cg : 1.0;
            const double m = __dmul_rn(a, b);
            ok = fabs(m) <= 1.5;
            s_fm[lane] = limbs(ok ? __double2ll_rn(m * 0x1p59) : 0);
          } else if (lane < 12) {
            const double t = lane == 9 ? p.cx + f.dx : lane == 10 ? p.cy + f.dy : p.cz + f.dz;
            ok = fabs(t) < 4000.0;
            const long long v = ok ? __double2ll_rn(t * 0x1p51) - p.ofix[lane - 9] : 0;
            ok = ok && llabs(v) < static_cast<long long>(kFixFar * 0x1p51);
            s_ft[lane - 9] = v;
          }
          fix = __all_sync(kFull, ok);
          __syncwarp();
        }
#pragma unroll 1
        for (int s = 0; s < S; ++s) {
          const int j = ch * kChunk + s * 32 + lane;
          const bool on = j < p.nl;
          // (idle lanes: far from every receptor atom, including the padding at +1e9)
          float4 l = make_float4(-1.0e9f, -1.0e9f, -1.0e9f, 0.0f);
          int lt = 0;
          if (on) {
            if (fix) {
              const int4 xy = __ldg(&p.lig_fix[2 * j]), z = __ldg(&p.lig_fix[2 * j + 1]);
              l.x = fix_float(rotate(s_fm[0], s_fm[1], s_fm[2], xy, z) + s_ft[0]);
              l.y = fix_float(rotate(s_fm[3], s_fm[4], s_fm[5], xy, z) + s_ft[1]);
              l.z = fix_float(rotate(s_fm[6], s_fm[7], s_fm[8], xy, z) + s_ft[2]);
              l.w = __int_as_float(z.z);
              lt = z.w;
            } else {
              const float3 c = atom32(p, f, pose, j);
              l = make_float4(c.x, c.y, c.z, static_cast<float>(p.lig_rel[j].w));
              lt = p.lig_type[j];
            }
            if (!GD_DCHECK(bp.err, lt >= 0 && lt < p.nt, 6)) lt = 0;
          }
          s_lig[s * 32 + lane] = l;
          s_lt[s * 32 + lane] = static_cast<uint16_t>(lt);
          // bounding sphere of the slot's 32 atoms: with a rigid pose the
          // precomputed small enclosing sphere moved with it (s_ssph, smaller
          // than the centroid's sphere), else the centroid's of these atoms
          const unsigned on_mask = __ballot_sync(kFull, on);
          float cx = 0.0f, cy = 0.0f, cz = 0.0f, rr = 0.0f;
          if (!cull) {
            cx = on ? l.x : 0.f, cy = on ? l.y : 0.f, cz = on ? l.z : 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
              cx += __shfl_xor_sync(kFull, cx, o);
              cy += __shfl_xor_sync(kFull, cy, o);
              cz += __shfl_xor_sync(kFull, cz, o);
            }
            const float inv = on_mask ? 1.0f / static_cast<float>(__popc(on_mask)) : 0.0f;
            cx *= inv;
            cy *= inv;
            cz *= inv;
            rr = on ? sqrtf((l.x - cx) * (l.x - cx) + (l.y - cy) * (l.y - cy) + (l.z - cz) * (l.z - cz))
                    : 0.0f;
            rr = warp_max(rr);
          }
          // axis-aligned bounding box of the same atoms (half-widths widened
          // like the radius so that FP32 rounding never shrinks it)
          const float lo_x = warp_min(on ? l.x : 3.0e38f), lo_y = warp_min(on ? l.y : 3.0e38f),
                      lo_z = warp_min(on ? l.z : 3.0e38f);
          const float hi_x = warp_max(on ? l.x : -3.0e38f), hi_y = warp_max(on ? l.y : -3.0e38f),
                      hi_z = warp_max(on ? l.z : -3.0e38f);
          if (lane == 0) {
            s_blob[s] = !on_mask ? make_float4(0.0f, 0.0f, 0.0f, -1.0e30f)
                                 : (cull ? s_ssph[s] : make_float4(cx, cy, cz, rr * 1.0001f + 0.01f));
            if (on_mask) {
              s_box[2 * s] = make_float4(0.5f * (lo_x + hi_x), 0.5f * (lo_y + hi_y), 0.5f * (lo_z + hi_z),
                                         0.5f * (hi_x - lo_x) * 1.0001f + 0.01f);
              s_box[2 * s + 1] = make_float4(0.5f * (hi_y - lo_y) * 1.0001f + 0.01f,
                                             0.5f * (hi_z - lo_z) * 1.0001f + 0.01f, 0.0f, 0.0f);
            } else {
              s_box[2 * s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
              s_box[2 * s + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
          }
        }
        __syncwarp();
        // phase-1 role of this lane: row (slot my_s, atom my_a of each 8-atom round)
        const float4 myb = my_s < S ? s_blob[my_s] : make_float4(0.0f, 0.0f, 0.0f, -1.0e30f);
        const float mlim = myb.w + reach;
        const float mlim2 = (myb.w >= 0.0f) ? mlim * mlim : -1.0f;  // empty slot: no row kept
        const float mnear = myb.w + reach_v, mnear2 = mnear * mnear;
        const float4 bx0 = s_box[2 * (my_s & (kMaxS - 1))], bx1 = s_box[2 * (my_s & (kMaxS - 1)) + 1];
        // per segment: flagged steps (high 16 bits) and recorded ones (low 16)
        int seg_cnt = 0;
        for (int kk = 0; kk < nk; ++kk, ++q) {
          const int g = seg_at(kk);
          const int st = static_cast<int>(q % kWS);
          const bool ok = __all_sync(kFull, mbar_wait(&s_bar[st], static_cast<uint32_t>((q / kWS) & 1)));
          if (!ok) {
            failed = true;
            break;
          }
          const int gbase = g * kSeg;
          const int na = min(kSeg, p.nr - gbase);
          const int sbase = st * kSeg;

          // Phase 1: lane (slot, atom) tests one row against the slot's sphere.
          // Kept rows go to the slot's list: far rows (Coulomb only) from the
          // front, near rows from the back; each run is padded with the far
          // dummy atom to whole steps.
          int nf_mine = 0, nn_mine = 0;  // far / near rows of this lane's slot
          uint32_t *my_list = s_list + my_s * kList;
          for (int b0 = 0; b0 < na; b0 += kBlk) {
            const float4 ra = s_pos[sbase + b0 + my_a];  // atoms past nr are padding far away
            const float dx = ra.x - myb.x, dy = ra.y - myb.y, dz = ra.z - myb.z;
            const float dc2 = dx * dx + dy * dy + dz * dz;
            // distance from the atom to the slot's box: a second lower bound on
            // every pair distance of the row (either bound may drop the row or
            // make it far)
            const float ex = fmaxf(fabsf(ra.x - bx0.x) - bx0.w, 0.0f), ey = fmaxf(fabsf(ra.y - bx0.y) - bx1.x, 0.0f),
                        ez = fmaxf(fabsf(ra.z - bx0.z) - bx1.y, 0.0f);
            const float db2 = ex * ex + ey * ey + ez * ez;
            const bool keep = dc2 < mlim2 && db2 < reach2, nearr = dc2 < mnear2 && db2 < reach_v2;
            const unsigned Mf = __ballot_sync(kFull, keep && !nearr), Mn = __ballot_sync(kFull, keep && nearr);
            const int at = sbase + b0 + my_a;
            const uint32_t idx = (pos_at + static_cast<uint32_t>(at) * 16) << 12 | static_cast<uint32_t>(s_meta[at].x);
            // at most na <= kSeg rows per slot: far rows fill [0, nf), near rows
            // (kList - nn, kList - 1], with room for both paddings in between
            const int pf = nf_mine + __popc(Mf & my_group & lt_mask), pn = kList - 1 - nn_mine - __popc(Mn & my_group & lt_mask);
            if (keep && !nearr && GD_DCHECK(bp.err, pf >= 0 && pf < kList, 1)) my_list[pf] = idx;
            if (keep && nearr && GD_DCHECK(bp.err, pn >= 0 && pn < kList, 2)) my_list[pn] = idx;

            nf_mine += __popc(Mf & my_group);
            nn_mine += __popc(Mn & my_group);
          }
          if (my_s < S && my_a < kAtoms &&
              GD_DCHECK(bp.err, nf_mine + my_a < kList && kList - 1 - nn_mine - my_a >= 0, 3)) {
            my_list[nf_mine + my_a] = far_row;
            my_list[kList - 1 - nn_mine - my_a] = far_row;
          }
          __syncwarp();

          // Phase 2: every term of the kept rows, kAtoms rows per step (two in
          // the last one where two are left: a run of 13 rows wastes one, not
          // three)
          float av = 0.0f, ae = 0.0f;  // ae: corrections from exact re-decisions (charge included)
#pragma unroll 1
          for (int s = 0; s < S; ++s) {
            const int nf = __shfl_sync(kFull, nf_mine, s * 8), nn = __shfl_sync(kFull, nn_mine, s * 8);
            const uint32_t *lst = s_list + s * kList;
            const float4 l = s_lig[s * 32 + lane];
            const float2 *tabl = tab + s_lt[s * 32 + lane];
            const int lser = SERIAL && ch * kChunk + s * 32 + lane < p.nl ? p.lig_serial[ch * kChunk + s * 32 + lane] : 0;
            float aes = 0.0f;  // sum of q_r / d2 over this slot's kept pairs
            int lc = 0;        // the lane's pairs within 8 A
            auto row = [&](uint32_t e) {
              if (!GD_DCHECK(bp.err, entry_atom(e) >= 0 && entry_atom(e) <= kFar, 4)) e = far_row;
              float4 r;
              asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                           : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
                           : "r"(e >> 12));
              return r;
            };
            // N consecutive entries in one load (N = 4: k0 is a multiple of 4, N = 2: even)
            auto entries = [&](int k0, uint32_t *e, auto count) {
              constexpr int N = decltype(count)::value;
              if constexpr (N == 4) {
                const uint4 v = *reinterpret_cast<const uint4 *>(lst + k0);
                e[0] = v.x;
                e[1] = v.y;
                e[2] = v.z;
                e[3] = v.w;
              } else if constexpr (N == 2) {
                const uint2 v = *reinterpret_cast<const uint2 *>(lst + k0);
                e[0] = v.x;
                e[1] = v.y;
              } else {
                e[0] = lst[k0];
              }
            };
            auto flag = [&](bool amb, int k0, int rows) {
              if (!__any_sync(kFull, amb)) return;
              if (lane == 0 && GD_DCHECK(bp.err, (seg_cnt >> 16) < kMaxS * (kList / kAtoms + 2), 7))
                s_fixq[seg_cnt >> 16] = static_cast<uint16_t>(k0 | s << 8 | rows << 12);
              seg_cnt += 1 << 16;
            };
            // far rows: Coulomb only.  Every FP32 d2 of a far row exceeds 144,
            // where d2 - 225 is exact (Sterbenz) and d2 < 225 is the whole
            // decision: one bound, one band.
            auto far_step = [&](int k0, auto count) {
              constexpr int N = decltype(count)::value;
              uint32_t e[N];
              entries(k0, e, count);
              bool amb = false;
#pragma unroll
              for (int i = 0; i < N; ++i) {
                const float4 r = row(e[i]);
                const float d2 = d2f(r, l.x, l.y, l.z), tf = __fsub_rn(d2, 225.0f);
                fma_if_lt0(aes, tf, r.w, rcp_approx(d2));
                amb = amb | (fabsf(tf) < ge);
              }
              flag(amb, k0, N);
            };
            // near rows: every term
            auto near_step = [&](int k0, auto count) {
              constexpr int N = decltype(count)::value;
              uint32_t e[N];
              entries(k0, e, count);
              bool amb = false, in[N], any_in = false;
#pragma unroll
              for (int i = 0; i < N; ++i) {
                const float4 r = row(e[i]);
                uint32_t rt = e[i] & 0xfffu;
                if (!GD_DCHECK(bp.err, static_cast<int>(rt) + s_lt[s * 32 + lane] < p.nt * p.nt, 5)) rt = 0;
                const float2 tp = __ldg(tabl + rt);
                const float d2 = d2f(r, l.x, l.y, l.z);
                const bool same = SERIAL && s_meta[entry_atom(e[i])].y == lser;
                pair32<SERIAL, CLAMP>(d2, r.w, tp, same, gv, ge, gdd, av, aes, amb);
                in[i] = d2 < 64.0f;
                any_in = any_in || in[i];
              }
              flag(amb, k0, N);
              // burial: a step with no pair within 8 A (about half of them)
              // has nothing to count; else the rows' ballots are recorded here
              // and added up once per segment (below)
              if (__any_sync(kFull, any_in)) {
                const int at = (seg_cnt & 0xffff) * kAtoms;
#pragma unroll
                for (int i = 0; i < N; ++i) {
                  const unsigned bm = __ballot_sync(kFull, in[i]);
                  lc += in[i];
                  if (lane == i && GD_DCHECK(bp.err, at + i < kMaxS * kList, 8)) s_cmask[at + i] = bm;
                }
                if (lane == 0) s_cstep[seg_cnt & 0xffff] = static_cast<uint16_t>(k0 | s << 8 | N << 12);
                ++seg_cnt;
              }
            };
            using Step = std::integral_constant<int, kAtoms>;
            using Two = std::integral_constant<int, 2>;
            int k0 = 0;
#pragma unroll 1
            for (; nf - k0 > (kAtoms == 4 ? 2 : 0); k0 += kAtoms) far_step(k0, Step());
            if (kAtoms == 4 && k0 < nf) far_step(k0, Two());
            // the first near step starts in the padding
            k0 = kList - (nn + kAtoms - 1) / kAtoms * kAtoms;
            if (kAtoms == 4 && ((nn - 1) & 2) == 0 && nn > 0) {  // one or two rows over
              near_step(k0 + 2, Two());
              k0 += 4;
            }
#pragma unroll 1
            for (; k0 < kList; k0 += kAtoms) near_step(k0, Step());
            ae = __fmaf_rn(aes, l.w, ae);
            if (lc) s_lcnt[s * 32 + lane] += lc;
          }
          __syncwarp();
          // exact re-decisions of the flagged steps' pairs in the guard band
          const int nfix = seg_cnt >> 16, ncs = seg_cnt & 0xffff;
#pragma unroll 1
          for (int t = 0; t < nfix; ++t) {
            const int e = s_fixq[t], k0 = e & 255, s = (e >> 8) & 15, rows = e >> 12;
            const int j = ch * kChunk + s * 32 + lane;
            if (j >= p.nl) continue;
            const float4 l = s_lig[s * 32 + lane];
#pragma unroll 1
            for (int i = 0; i < rows; ++i) {
              const int ixi = entry_atom(s_list[s * kList + k0 + i]);
              if (ixi == kFar || !GD_DCHECK(bp.err, ixi >= 0 && ixi < kFar, 4)) continue;
              const float4 ri = s_pos[ixi];
              if (!near_band(d2f(ri, l.x, l.y, l.z), gv, ge, gdd)) continue;
              const int2 mt = s_meta[ixi];
              const FixOut fo = fix_pair<SERIAL, CLAMP>(p, f, pose, j, fix && p.fix, s_fm, s_ft, ri, gbase + ixi - sbase, mt.x, mt.y, l.x, l.y, l.z, l.w,
                                                        s_lt[s * 32 + lane], SERIAL ? p.lig_serial[j] : 0);
              av += fo.dv;
              ae += fo.de;
              if (fo.dl) {
                s_lcnt[s * 32 + lane] += fo.dl;
                atomicAdd(&s_rc[ixi - sbase], fo.dl);
              }
            }
          }
          // receptor burial counts of the near rows (the far atom's ballots are 0)
          for (int t = lane; t < ncs * kAtoms; t += 32) {
            const int e = s_cstep[t / kAtoms], i = t % kAtoms;
            const unsigned bm = i < (e >> 12) ? s_cmask[t] : 0u;
            if (bm)
              atomicAdd(&s_rc[entry_atom(s_list[((e >> 8) & 15) * kList + (e & 255) + i]) - sbase], __popc(bm));
          }
          seg_cnt = 0;
          fv += fx_energy(av, bp.err);
          fe += fx_energy(ae, bp.err);
          __syncwarp();
          // receptor burial counts of this segment into the per-item counters
          for (int i = lane; i < na; i += 32) {
            const int c = s_rc[i];
            if (c) {
              if (SPLIT) {
                // a count never exceeds the ligand's atoms (< 65,536 in split
                // launches), so the two halves of a word never carry into each other
                const int a = gbase + i;
                if (GD_DCHECK(bp.err, a < bp.max_nr, 10))
                  atomicAdd(&bp.pcount[static_cast<size_t>(gp) * ((bp.max_nr + 1) >> 1) + (a >> 1)],
                            static_cast<unsigned>(c) << ((a & 1) * 16));
              }
              else bump_count(cnt, gbase + i, c);
              s_rc[i] = 0;
            }
          }
          __syncwarp();
          if (lane == 0 && kk + kWS < nk) {
            issue_seg(q + kWS, seg_at(kk + kWS), p, s_pos, s_meta, s_bar);
            q_issued = q + kWS + 1;
          }
        }
      }
      if (failed) break;
      __syncwarp();
      // the chunk's per-lane partials (split and whole-pose items add them
      // alike, so both give bit-identical energies): ligand desolvation from
      // this chunk's burial counts; with receptor parts the counts are only
      // partial here and go to the pose's counters
      double dch = 0.0;
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const int lcnt = s_lcnt[s * 32 + lane], j = ch * kChunk + s * 32 + lane;
        if (R == 1) {
          if (j < p.nl) dch += p.lig_desolv[static_cast<size_t>(j) * 11 + min(lcnt, 10)];
        } else if (j < p.nl && lcnt != 0 && GD_DCHECK(bp.err, j < bp.max_nl, 11)) {
          atomicAdd(&bp.lcount[static_cast<size_t>(gp) * bp.max_nl + j], static_cast<unsigned>(lcnt));
        }
      }
      if (SPLIT) {
        const int slot = ch * R + rpart;
        if (!GD_DCHECK(bp.err, slot < bp.max_chunks, 9)) break;
        double *pt = bp.part + (static_cast<size_t>(gp) * bp.max_chunks + slot) * 96;
        reinterpret_cast<long long *>(pt)[lane] = fv;
        reinterpret_cast<long long *>(pt)[32 + lane] = fe;
        pt[64 + lane] = dch;
        if (SPLIT == 2 && rem == 0) {
          // with receptor parts the pose's first item adds its restraint
          // energy, beside other items' pairs and not at the end of the launch
          // (one pose of 2,538 x 1,280 atoms 95 -> 91 us; 65,536 in chunks
          // alone were 0.8 % slower with it)
          double air;
          int sat;
          warp_air(p, f, pose, lane, air, sat);
          if (lane == 0) bp.air[gp] = make_double2(air, static_cast<double>(sat));
        }
      } else {
        vdw_i += fv;
        elec_i += fe;
        desolv_t += dch;
      }
    }
    if (failed) {
      // a bulk copy did not land in time: record it, wait (bounded) for the
      // copies this warp still has in flight, and stop this warp
      if (lane == 0) {
        atomicExch(bp.err, kDevTimeout);
        for (long long u = q; u < q_issued; ++u) mbar_wait(&s_bar[u % kWS], static_cast<uint32_t>((u / kWS) & 1));
      }
      __syncwarp();
      return;
    }
    if (SPLIT) {
      // publish this chunk; the warp that completes the pose reduces it
      __threadfence();
      __syncwarp();
      int done = 0;
      if (lane == 0) done = atomicAdd(&bp.pdone[gp], 1);
      done = __shfl_sync(kFull, done, 0);
      if (done != per_pose - 1) continue;
      __threadfence();
      if constexpr (SPLIT == 2) {
        // every loop here waits for L2 once or twice per round; with receptor
        // parts (launches of few poses) nothing runs beside the last poses'
        // rounds, so theirs hold more loads: one pose of 6,800 x 2,500 atoms 151 ->
        // 139 us.  The sums keep their order.
        constexpr int kP = 8, kC = 3, kR = 16;
        const double *pose_part = bp.part + static_cast<size_t>(gp) * bp.max_chunks * 96;
        for (int c0 = 0; c0 < per_pose; c0 += kP) {
          long long v[kP], e[kP];
#pragma unroll
          for (int u = 0; u < kP; ++u) {
            const long long *pi = reinterpret_cast<const long long *>(pose_part + min(c0 + u, per_pose - 1) * 96);
            v[u] = __ldcg(pi + lane);
            e[u] = __ldcg(pi + 32 + lane);
          }
#pragma unroll
          for (int u = 0; u < kP; ++u) {
            if (c0 + u < per_pose) {
              vdw_i += v[u];
              elec_i += e[u];
            }
          }
        }
        // ligand desolvation chunk by chunk, in the same order and arithmetic
        // as whole-pose items
        for (int c0 = 0; c0 < nchunks; c0 += kC) {
          unsigned n[kC * S];
          double t[kC * S];
#pragma unroll
          for (int u = 0; u < kC * S; ++u) {
            const int j = c0 * kChunk + u * 32 + lane;
            n[u] = j < p.nl ? __ldcg(&bp.lcount[static_cast<size_t>(gp) * bp.max_nl + j]) : 0u;
          }
#pragma unroll
          for (int u = 0; u < kC * S; ++u) {
            const int j = c0 * kChunk + u * 32 + lane;
            t[u] = j < p.nl ? p.lig_desolv[static_cast<size_t>(j) * 11 + (n[u] < 10u ? n[u] : 10u)] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < kC; ++u) {
            double dc = 0.0;
#pragma unroll
            for (int s = 0; s < S; ++s) dc += t[u * S + s];
            if (c0 + u < nchunks) desolv_t += dc;
          }
        }
        for (int i0 = 0; i0 < p.nr; i0 += 32 * kR) {
          unsigned w[kR];
          double t[kR];
#pragma unroll
          for (int u = 0; u < kR; ++u) {
            const int i = i0 + u * 32 + lane;
            w[u] = i < p.nr ? __ldcg(&bp.pcount[static_cast<size_t>(gp) * ((bp.max_nr + 1) >> 1) + (i >> 1)]) : 0u;
          }
#pragma unroll
          for (int u = 0; u < kR; ++u) {
            const int i = i0 + u * 32 + lane;
            const unsigned c = (w[u] >> ((lane & 1) * 16)) & 0xffffu;
            t[u] = i < p.nr ? p.rec_desolv[static_cast<size_t>(i) * 11 + (c < 10u ? c : 10u)] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < kR; ++u) desolv_t += t[u];
        }
      } else {
        for (int c = 0; c < per_pose; ++c) {
          const long long *pi =
              reinterpret_cast<const long long *>(bp.part + (static_cast<size_t>(gp) * bp.max_chunks + c) * 96);
          vdw_i += __ldcg(pi + lane);
          elec_i += __ldcg(pi + 32 + lane);
        }
        for (int c = 0; c < nchunks; ++c)
          desolv_t += __ldcg(bp.part + (static_cast<size_t>(gp) * bp.max_chunks + c) * 96 + 64 + lane);
        // four rounds' loads in flight, added in order
        for (int i0 = 0; i0 < p.nr; i0 += 128) {
          double t[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * 32 + lane;
            t[u] = 0.0;
            if (i < p.nr) {
              const unsigned w = __ldcg(&bp.pcount[static_cast<size_t>(gp) * ((bp.max_nr + 1) >> 1) + (i >> 1)]);
              const unsigned c = (w >> ((i & 1) * 16)) & 0xffffu;
              t[u] = p.rec_desolv[static_cast<size_t>(i) * 11 + (c < 10u ? c : 10u)];
            }
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) desolv_t += t[u];
        }
      }
    } else {
      // receptor burial -> desolvation; reset the counters for the next item
      for (int i = lane; i < p.nr; i += 32) {
        const int c = cnt[i];
        desolv_t += p.rec_desolv[static_cast<size_t>(i) * 11 + (c < 10 ? c : 10)];
        cnt[i] = 0;
      }
    }
    const double vdw_t = static_cast<double>(warp_sum_ll(vdw_i)) * 0x1p-32;
    const double elec_t = static_cast<double>(warp_sum_ll(elec_i)) * 0x1p-32;
    desolv_t = warp_sum(desolv_t);
    double air;
    int sat;
    if (SPLIT == 2) {
      const double2 a = __ldcg(&bp.air[gp]);
      air = a.x;
      sat = static_cast<int>(a.y);
    } else {
      warp_air(p, f, pose, lane, air, sat);
    }
    if (lane == 0) write_pose(p, pose, vdw_t, elec_t, desolv_t, air, sat);
    __syncwarp();
  }
}

// Split-mode kernel (a work item is one ligand chunk of a pose): one variant,
// 4 slots and 4 rows per step, five CTAs per SM, used for launches with few
// poses per warp.
constexpr int kSplitTune = -1;
constexpr int kSplitPartsTune = -2;  // the split kernel with receptor parts

// Kernel variants.  The common case (no equal receptor/ligand serials, no
// clamp needed) has a tuning grid of slots per lane S, receptor atoms per
// inner step A and minimum CTAs per SM (register cap); the rare cases run
// one variant.  The tuning value encodes S + 16 (A = 2) or + 64 (A = 4),
// + 256 for the register cap of five resident CTAs per SM.
template <typename F>
cudaError_t with_variant(int tune, bool serial, bool clamp, F f) {
  if (tune == kSplitTune) return serial ? f(k_score_f32w<4, 4, 5, true, false, 1>) : f(k_score_f32w<4, 4, 5, false, false, 1>);
  if (tune == kSplitPartsTune)
    return serial ? f(k_score_f32w<4, 4, 5, true, false, 2>) : f(k_score_f32w<4, 4, 5, false, false, 2>);
  if (serial || clamp) {
    if (serial && clamp) return f(k_score_f32w<4, 1, 4, true, true, 0>);
    if (serial) return f(k_score_f32w<4, 1, 4, true, false, 0>);
    return f(k_score_f32w<4, 1, 4, false, true, 0>);
  }
  switch (tune) {
    case 4: return f(k_score_f32w<4, 1, 4, false, false, 0>);
    case 64 + 2: return f(k_score_f32w<2, 4, 4, false, false, 0>);
    case 64 + 4: return f(k_score_f32w<4, 4, 4, false, false, 0>);
    case 256 + 64 + 2: return f(k_score_f32w<2, 4, 5, false, false, 0>);
    case 16 + 4: return f(k_score_f32w<4, 2, 4, false, false, 0>);
    default: return f(k_score_f32w<4, 4, 5, false, false, 0>);  // 256 + 64 + 4 = kDefaultF32Tune
  }
}

// Rows per step of a variant.
int variant_atoms(int tune, bool serial, bool clamp) {
  if (tune == kSplitTune || tune == kSplitPartsTune) return 4;
  if (serial || clamp || tune == 4) return 1;
  return tune == 16 + 4 ? 2 : 4;
}

// The dynamic shared memory of a CTA can exceed the 48 KB default (receptors
// near kCntSmemMax keep their burial counters there): the kernel's limit is
// raised before the occupancy query, which otherwise reports an invalid
// configuration.
cudaError_t occupancy_var(int tune, bool serial, bool clamp, size_t smem, int *per_sm) {
  return with_variant(tune, serial, clamp, [&](auto kern) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kern, kWarps * 32, smem);
  });
}

cudaError_t launch_var(int tune, const BatchParams &bp, bool serial, bool clamp, size_t smem, int grid,
                       cudaStream_t st) {
  return with_variant(tune, serial, clamp, [&](auto kern) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    kern<<<grid, kWarps * 32, smem, st>>>(bp);
    return cudaGetLastError();
  });
}

}  // namespace

// Work items are taken from the queue in descriptor order: put the complexes
// with the costliest poses first so that the last items of a launch are the
// cheap ones (longest-processing-time-first).
static std::vector<ScoreParams> lpt_order(const std::vector<ScoreParams> &descs) {
  std::vector<ScoreParams> v = descs;
  std::stable_sort(v.begin(), v.end(), [](const ScoreParams &a, const ScoreParams &b) {
    return static_cast<long long>(a.nr) * a.nl > static_cast<long long>(b.nr) * b.nl;
  });
  return v;
}

// Launch geometry of a batch: slots per lane, shared memory, grid.
struct BatchPlan {
  int tune, smem_cnt, max_nr, grid;
  size_t smem;
  std::vector<long long> start;       // work-item prefix per complex
  std::vector<long long> pose_start;  // pose prefix per complex
  int split = 0, max_chunks = 1;
  int rparts = 1, max_nl = 0;  // receptor parts per chunk (split mode), longest ligand
  size_t part_b = 0, cnt_b = 0, done_b = 0, lcnt_b = 0, air_b = 0;  // split-mode scratch
};

constexpr size_t kSplitScratchMax = size_t(4) << 30;  // split scratch beyond this: whole poses
constexpr int kMaxRparts = 24;  // receptor parts per chunk, at most (GD_TUNE_RPARTS accepts 1..8)

static size_t al256(size_t b) { return (b + 255) / 256 * 256; }

// Work items are the ligand chunks of the poses (split mode) whenever the
// split scratch fits (4 GiB and the context's HBM budget): no warp waits on a
// long pose at the end of a launch, which matters most with few poses per
// warp (one GA generation of a few jobs, one docking run's population, a few
// thousand poses of a large complex) and was measured no slower with many.
// Whole poses per item otherwise, and where well depths need the clamp; the
// energies are bit-identical either way.  Molecules that share serial numbers,
// as in two separate files, have split kernels of their own: in whole poses a
// pair of 2,538 x 1,280 atoms took 5.7 ms for one pose and 7.3 for 150, in
// chunks 0.10 and 0.40.
static gd_status plan_batch(gd_context *ctx, const std::vector<ScoreParams> &descs, bool serial, bool clamp,
                            int slots, bool allow_split, BatchPlan *pl) {
  const int ncx = static_cast<int>(descs.size());
  const int chunk_split = 32 * 4;  // the split kernel's chunk of ligand atoms
  pl->start.assign(ncx + 1, 0);
  pl->pose_start.assign(ncx + 1, 0);
  pl->max_nr = 0;
  pl->max_nl = 0;
  pl->max_chunks = 1;
  long long chunk_items = 0;  // (pose, chunk) items of a split launch
  int max_nseg = 1;
  for (int c = 0; c < ncx; ++c) {
    pl->pose_start[c + 1] = pl->pose_start[c] + descs[c].n_poses;
    pl->max_nr = std::max(pl->max_nr, descs[c].nr);
    pl->max_nl = std::max(pl->max_nl, descs[c].nl);
    const int nch = std::max(1, (descs[c].nl + chunk_split - 1) / chunk_split);
    pl->max_chunks = std::max(pl->max_chunks, nch);
    chunk_items += static_cast<long long>(descs[c].n_poses) * nch;
    max_nseg = std::max(max_nseg, (descs[c].nr + kSeg - 1) / kSeg);
  }
  const long long poses = pl->pose_start[ncx];
  pl->tune = slots;
  auto fit = [&](int smem_cnt, int *per_sm) -> cudaError_t {
    pl->smem_cnt = smem_cnt;
    pl->smem = warp_layout(smem_cnt, variant_atoms(pl->tune, serial, clamp)).total * kWarps;
    cudaError_t e = occupancy_var(pl->tune, serial, clamp, pl->smem, per_sm);
    if (e == cudaSuccess && *per_sm < 1) e = cudaErrorInvalidConfiguration;
    return e;
  };
  int per_sm = 0;
  cudaError_t e = fit(pl->max_nr <= kCntSmemMax ? ((pl->max_nr + 15) / 16) * 16 : 0, &per_sm);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "batched scoring occupancy");
  // receptor parts: R interleaved segment sets of each chunk, so that the SMs
  // fill and the last items to finish are short.  A part's item pays the
  // chunk's set-up again, and a receptor of g segments spreads that over
  // about g/R segments, so R falls with the launch's rounds (items per
  // resident warp, w) and grows with g: R = 1 + 0.75 sqrt(g) / w, rounded.
  // The best R of 1..8, measured on receptors of 4 to 107 segments at w of
  // 0.1 to 50, lies within one of it; R = 1 starts at w of 10 for 40
  // segments, where both cost the same (4,800 poses: 6.51 and 6.50 ms; 1,200
  // poses: 1.98 ms at R = 1, 1.83 at 3).  From 8 parts on more of them pay
  // only in launches of a fraction of a round (one pose of 2,538 x 1,280
  // atoms: 135 us at 8, 114 at 24; 150 poses: 371 at 8, 381 at 16), so there
  // the slope is an eighth.  GD_TUNE_RPARTS forces R.  The energies do not
  // depend on R (fixed-point sums).
  int split_per_sm = 0;
  {
    const int keep_tune = pl->tune;
    pl->tune = kSplitTune;
    e = fit(0, &split_per_sm);
    pl->tune = keep_tune;
    if (e != cudaSuccess) return cuda_fail(ctx, e, "batched scoring occupancy");
    e = fit(pl->max_nr <= kCntSmemMax ? ((pl->max_nr + 15) / 16) * 16 : 0, &per_sm);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "batched scoring occupancy");
  }
  int R = ctx->tune_rparts;
  if (R <= 0) {
    const double rounds = static_cast<double>(std::max(chunk_items, 1LL)) / split_per_sm / kWarps / ctx->sm_count;
    const double want = 1.5 + 0.75 * std::sqrt(static_cast<double>(max_nseg)) / rounds;
    R = static_cast<int>(std::min({want, 7.0 + want / 8.0, static_cast<double>(std::max(1, std::min(kMaxRparts, max_nseg)))}));
  }
  auto split_bytes = [&](int r, size_t *part_b, size_t *cnt_b, size_t *lcnt_b) {
    *part_b = static_cast<size_t>(poses) * pl->max_chunks * r * 96 * sizeof(double);
    *cnt_b = static_cast<size_t>(poses) * ((pl->max_nr + 1) / 2) * sizeof(unsigned);
    *lcnt_b = r > 1 ? static_cast<size_t>(poses) * std::max(pl->max_nl, 1) * sizeof(unsigned) : 0;
    const size_t b = al256(*part_b) + al256(*cnt_b) + al256(static_cast<size_t>(poses) * sizeof(int)) + al256(*lcnt_b) +
                     (r > 1 ? al256(static_cast<size_t>(poses) * sizeof(double2)) : 0);
    // (further parts leave half of what a budget has left)
    const uint64_t left = ctx->budget == 0 ? UINT64_MAX : ctx->budget > ctx->in_use ? ctx->budget - ctx->in_use : 0;
    return b <= kSplitScratchMax && b <= (r > 1 ? left / 2 : left);
  };
  size_t part_b = 0, cnt_b = 0, lcnt_b = 0;
  bool fits = split_bytes(R, &part_b, &cnt_b, &lcnt_b);
  while (!fits && R > 1 && ctx->tune_rparts <= 0) {
    R /= 2;
    fits = split_bytes(R, &part_b, &cnt_b, &lcnt_b);
  }
  pl->split = 0;
  // split launches keep receptor burial counts in 16 bits: ligands up to 65,535 atoms
  if (allow_split && fits && poses > 0 && (pl->max_chunks > 1 || R > 1) && !clamp && pl->max_nl < 65536)
    pl->split = ctx->tune_split != 1;
  if (pl->split) {
    pl->rparts = R;
    pl->part_b = part_b;
    pl->cnt_b = cnt_b;
    pl->lcnt_b = lcnt_b;
    pl->done_b = static_cast<size_t>(poses) * sizeof(int);
    pl->air_b = R > 1 ? static_cast<size_t>(poses) * sizeof(double2) : 0;
    pl->tune = R > 1 ? kSplitPartsTune : kSplitTune;
    e = fit(0, &per_sm);  // burial counters live in the split scratch
    if (e != cudaSuccess) return cuda_fail(ctx, e, "batched scoring occupancy");
  } else {
    pl->rparts = 1;
    pl->part_b = pl->cnt_b = pl->done_b = pl->lcnt_b = pl->air_b = 0;
  }
  for (int c = 0; c < ncx; ++c) {
    const long long per_pose =
        pl->split ? static_cast<long long>(std::max(1, (descs[c].nl + chunk_split - 1) / chunk_split)) * pl->rparts : 1;
    pl->start[c + 1] = pl->start[c] + static_cast<long long>(descs[c].n_poses) * per_pose;
  }
  const long long items = pl->start[ncx];
  pl->grid = static_cast<int>(std::max<long long>(
      1, std::min<long long>((items + kWarps - 1) / kWarps, static_cast<long long>(per_sm) * ctx->sm_count)));
  return GD_OK;
}

// Layout of the argument block: descriptors, item prefix, work counter, pose
// prefix, per-warp global burial counters (large receptors, whole-pose
// items), split-mode partials, receptor burial counts, item counters and
// (receptor parts) ligand burial counts.
struct ArgLayout {
  size_t desc, start, queue, pstart, gcounts, part, air, pcount, pdone, lcount, total;
};

static ArgLayout arg_layout(int ncx, const BatchPlan &pl, size_t gcount_bytes) {
  ArgLayout L{};
  size_t o = 0;
  L.desc = o;
  o += al256(sizeof(ScoreParams) * ncx);
  L.start = o;
  o += al256(sizeof(long long) * (ncx + 1));
  L.pstart = o;
  o += al256(sizeof(long long) * (ncx + 1));
  L.gcounts = o;
  o += al256(gcount_bytes);
  L.part = o;
  o += al256(pl.part_b);
  L.air = o;
  o += al256(pl.air_b);
  L.queue = o;  // from here on cleared before every launch
  o += al256(sizeof(unsigned long long));
  L.pcount = o;
  o += al256(pl.cnt_b);
  L.pdone = o;
  o += al256(pl.done_b);
  L.lcount = o;
  o += al256(pl.lcnt_b);
  L.total = o;
  return L;
}

static size_t gcount_stride(const BatchPlan &pl) {
  return (pl.smem_cnt || pl.split) ? 0 : ((pl.max_nr + 127) / 128) * 128;
}

static gd_status upload_args(gd_context *ctx, const std::vector<ScoreParams> &descs, const BatchPlan &pl,
                             const ArgLayout &L, char *arg, cudaStream_t stream, bool sync) {
  const int ncx = static_cast<int>(descs.size());
  // staged from pageable memory: the copy has left the host buffer when the
  // call returns, so back-to-back launches cannot race on it
  std::vector<char> h(L.gcounts);
  std::memcpy(h.data() + L.desc, descs.data(), sizeof(ScoreParams) * ncx);
  std::memcpy(h.data() + L.start, pl.start.data(), sizeof(long long) * (ncx + 1));
  std::memcpy(h.data() + L.pstart, pl.pose_start.data(), sizeof(long long) * (ncx + 1));
  const cudaError_t e = sync ? cudaMemcpy(arg, h.data(), h.size(), cudaMemcpyHostToDevice)
                             : cudaMemcpyAsync(arg, h.data(), h.size(), cudaMemcpyHostToDevice, stream);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "batched scoring arguments");
  return GD_OK;
}

// Reset the work counter (and the split-mode counters) and launch.
static gd_status launch_args(gd_context *ctx, int ncx, const BatchPlan &pl, const ArgLayout &L, char *arg,
                             bool serial, bool clamp, cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(arg + L.queue, 0, pl.split ? L.total - L.queue : sizeof(unsigned long long), stream);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "batched scoring reset");
  BatchParams bp{};
  bp.descs = reinterpret_cast<const ScoreParams *>(arg + L.desc);
  bp.item_start = reinterpret_cast<const long long *>(arg + L.start);
  bp.ncx = ncx;
  bp.total = pl.start[ncx];
  bp.queue = reinterpret_cast<unsigned long long *>(arg + L.queue);
  const size_t gs = gcount_stride(pl);
  bp.gcounts = gs ? reinterpret_cast<uint8_t *>(arg + L.gcounts) : nullptr;
  bp.gcount_stride = static_cast<int>(gs);
  bp.smem_cnt = pl.smem_cnt;
  bp.max_nr = pl.max_nr;
  bp.err = ctx->d_err;
  bp.split = pl.split;
  bp.drop_copy = ctx->tune_fault == 1;
  bp.pose_start = reinterpret_cast<const long long *>(arg + L.pstart);
  bp.max_chunks = pl.max_chunks * pl.rparts;
  bp.part = pl.split ? reinterpret_cast<double *>(arg + L.part) : nullptr;
  bp.air = pl.split && pl.rparts > 1 ? reinterpret_cast<double2 *>(arg + L.air) : nullptr;
  bp.pcount = pl.split ? reinterpret_cast<unsigned *>(arg + L.pcount) : nullptr;
  bp.pdone = pl.split ? reinterpret_cast<int *>(arg + L.pdone) : nullptr;
  bp.rparts = pl.split ? pl.rparts : 1;
  bp.lcount = pl.split && pl.rparts > 1 ? reinterpret_cast<unsigned *>(arg + L.lcount) : nullptr;
  bp.max_nl = pl.max_nl;
  e = launch_var(pl.tune, bp, serial, clamp, pl.smem, pl.grid, stream);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "batched scoring launch");
  return GD_OK;
}

// Score the poses of several complexes in one persistent launch (FP32 form).
// descs[c] describes complex c with its frames/models, outputs and pose count.
gd_status launch_score_batch_f32(gd_context *ctx, const std::vector<ScoreParams> &descs_in, bool serial, bool clamp,
                                 int slots, cudaStream_t stream) {
  const std::vector<ScoreParams> descs = lpt_order(descs_in);
  const int ncx = static_cast<int>(descs.size());
  if (ncx == 0) return GD_OK;
  BatchPlan pl;
  gd_status s = plan_batch(ctx, descs, serial, clamp, slots, true, &pl);
  if (s != GD_OK) return s;
  if (pl.start[ncx] == 0) return GD_OK;
  const ArgLayout L = arg_layout(ncx, pl, gcount_stride(pl) * static_cast<size_t>(pl.grid) * kWarps);
  s = ensure_batch_scratch(ctx, L.total);
  if (s != GD_OK) return s;
  char *arg = static_cast<char *>(ctx->d_batch);
  s = upload_args(ctx, descs, pl, L, arg, stream, false);
  if (s != GD_OK) return s;
  return launch_args(ctx, ncx, pl, L, arg, serial, clamp, stream);
}

// A batched scoring launch whose argument block is uploaded once and whose
// launch (counter resets + kernel) can be replayed, e.g. inside a captured
// CUDA graph.
struct BatchLaunch {
  BatchPlan plan;
  ArgLayout layout{};
  bool serial = false, clamp = false;
  char *d_arg = nullptr;
  int ncx = 0;
};

gd_status batch_prepare(gd_context *ctx, const std::vector<ScoreParams> &descs_in, bool serial, bool clamp, int slots,
                        BatchLaunch **out) {
  *out = nullptr;
  const std::vector<ScoreParams> descs = lpt_order(descs_in);
  BatchLaunch *b = new BatchLaunch();
  b->serial = serial;
  b->clamp = clamp;
  b->ncx = static_cast<int>(descs.size());
  gd_status s = plan_batch(ctx, descs, serial, clamp, slots, true, &b->plan);
  if (s != GD_OK) {
    delete b;
    return s;
  }
  b->layout = arg_layout(b->ncx, b->plan, gcount_stride(b->plan) * static_cast<size_t>(b->plan.grid) * kWarps);
  void *p = nullptr;
  s = dev_alloc(ctx, b->layout.total, &p);
  if (s != GD_OK) {
    delete b;
    return s;
  }
  b->d_arg = static_cast<char *>(p);
  s = upload_args(ctx, descs, b->plan, b->layout, b->d_arg, nullptr, true);
  if (s != GD_OK) {
    batch_free(ctx, b);
    return s;
  }
  *out = b;
  return GD_OK;
}

gd_status batch_launch(gd_context *ctx, BatchLaunch *b, cudaStream_t stream) {
  if (b->plan.start[b->ncx] == 0) return GD_OK;
  return launch_args(ctx, b->ncx, b->plan, b->layout, b->d_arg, b->serial, b->clamp, stream);
}

void batch_free(gd_context *ctx, BatchLaunch *b) {
  if (!b) return;
  if (b->d_arg) dev_free(ctx, b->d_arg, b->layout.total);
  delete b;
}

// ---------------------------------------------------------------------------
// Scoring without any device allocation.
//
// Some hosts of this library cannot allocate device memory once scoring
// starts: a docking service that hands the whole GPU to a pool allocator at
// start-up (a cudaMalloc from inside the scoring path would fail or fragment
// that pool), or a real-time host loop that forbids the unbounded latency of
// an allocation.  For them the FP32 scoring kernel can take its small argument
// block (complex descriptor, pose-count prefix sums, work counter) from the
// file-scope array below instead of from context scratch memory.  The array
// is kNoAllocScratchBytes bytes on every GPU that loads the library and stays
// allocated until the process exits.  In host code its name is only a
// stand-in: the device address is looked up once per device with
// cudaGetSymbolAddress while that device is current.
constexpr size_t kNoAllocScratchBytes = 4096;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
void *g_noalloc_addr[kMaxDevices] = {};

// Device address of g_noalloc_scratch on the current device (looked up on
// the first call for that device).
gd_status noalloc_scratch(gd_context *ctx, void **out) {
  if (ctx->device < 0 || ctx->device >= kMaxDevices) return fail(ctx, GD_ERR_INVALID_ARG, "device index too large");
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_addr[ctx->device]) {
    void *ptr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess || !ptr) return cuda_fail(ctx, e, "cudaGetSymbolAddress(no-allocation scratch)");
    g_noalloc_addr[ctx->device] = ptr;
  }
  *out = g_noalloc_addr[ctx->device];
  return GD_OK;
}
}  // namespace

}  // namespace gd

extern "C" gd_status gd_score_frames_device_noalloc(gd_complex *cx, const gd_pose_frame *d_frames, int32_t n,
                                                    double max_displacement, gd_pose_energy *d_out, void *stream) {
  using namespace gd;
  if (!cx) return GD_ERR_INVALID_ARG;
  gd_context *ctx = cx->ctx;
  if (n < 0 || (n > 0 && (!d_frames || !d_out))) return fail(ctx, GD_ERR_INVALID_ARG, "bad frames/out");
  if (!(max_displacement >= 0.0)) return fail(ctx, GD_ERR_INVALID_ARG, "bad max_displacement");
  if (cx->nr > kCntSmemMax)
    return fail(ctx, GD_ERR_INVALID_ARG,
                "receptor has " + std::to_string(cx->nr) + " atoms; scoring without allocation handles at most " +
                    std::to_string(kCntSmemMax));
  static_assert(4 * 256 + 2 * 256 + sizeof(ScoreParams) <= kNoAllocScratchBytes,
                "no-allocation scratch too small for one complex");
  if (n == 0) return GD_OK;
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaSetDevice");
  void *scratch = nullptr;
  gd_status s = noalloc_scratch(ctx, &scratch);
  if (s != GD_OK) return s;
  const std::vector<ScoreParams> descs{make_params(cx, d_frames, nullptr, n, d_out, max_displacement)};
  const int slots = ctx->tune_f32_slots ? ctx->tune_f32_slots : kDefaultF32Tune;
  BatchPlan pl;
  s = plan_batch(ctx, descs, cx->serial_overlap, cx->need_clamp, slots, false, &pl);
  if (s != GD_OK) return s;
  // whole-pose items with counters in shared memory (receptor <= kCntSmemMax
  // atoms): the argument block is all the scratch there is
  const ArgLayout L = arg_layout(1, pl, 0);
  if (L.total > kNoAllocScratchBytes) return fail(ctx, GD_ERR_STATE, "no-allocation scratch too small");
  cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : ctx->stream;
  char *arg = static_cast<char *>(scratch);
  s = upload_args(ctx, descs, pl, L, arg, st, false);
  if (s != GD_OK) return s;
  return launch_args(ctx, 1, pl, L, arg, cx->serial_overlap, cx->need_clamp, st);
}

