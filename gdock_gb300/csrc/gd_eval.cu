// Docking-quality metrics of poses against a reference ligand structure: the
// evaluator of gdock (src/evaluator.rs:50-186), used for the per-generation
// metrics report and as the debug fitness (src/chromosome.rs:93-106).
//
// Host (gd_evaluator_create), following src/evaluator.rs:50-66,170-186:
//   - interface residues: receptor and reference residues with an atom pair
//     at distance <= 5 A;
//   - receptor interface = receptor atoms of those residues, reference
//     interface likewise, native contacts = their atom pairs at <= 5 A,
//     identified by (chain, residue, atom name) on both sides;
//   - the per-pose work then needs, per ligand atom: its pairing in the
//     L-RMSD (zip of the ligand with the reference), its pairing in the
//     i-RMSD (zip of the ligand's interface-residue atoms with the reference
//     interface), and the receptor atoms whose contact with it has a native
//     identity (a docked contact counts once when it is native); ligand atoms
//     with none of these are left out.
// Device (k_dockq): the lanes of one warp (or of eight, for few poses) take a
// pose's ligand atoms; transform, distance and sums are fixed-point integers.
// Offsets from the rotation centre lie on a grid of 2^-50 A, positions of 2^-51,
// distances with a component from 64 A on of 2^-45: coarser than a double next to
// its own zero (offsets below 4 A, positions below 2 A), finer than what the
// transform's FP64 roundings leave of a position at a protein's size.  No rounding
// above 2^-51 A is shared by all atoms, so the metrics are closer to their exact
// values than in the reference's order (mean error of the RMSD of poses 0.5 to 10
// A off 4.8e-17 to 7.4e-17, in the reference's order 5.3e-17 to 8.8e-17).
// Contacts are decided in FP32 outside a guard band and exactly (the reference's
// transform and threshold) inside it, and distances that cancellation would spoil
// (below 1/4 A) or that leave the fixed-point range are formed in FP64 in the
// reference's order.
//   rmsd  = sqrt(sum over pairs of distance / |reference|)    (src/evaluator.rs:86-103;
//   irmsd = likewise over the interface pairings               the sum is of distances)
//   fnat  = docked native contacts / |native contacts|
//   dockq = (fnat + 1/(1 + (irmsd/1.5)^2) + 1/(1 + (rmsd/8.5)^2)) / 3
#include <algorithm>
#include <cmath>
#include <cstring>
#include <set>
#include <tuple>
#include <vector>

#include "gd_device.cuh"

struct Fix3 { long long x, y, z, pad; };

struct gd_evaluator {
  gd_complex *cx = nullptr;
  gd_context *ctx = nullptr;
  int n_u = 0;                            // ligand atoms the metrics read
  int n_ref = 0, n_iref = 0, n_native = 0;  // divisors: |reference|, |reference interface|, |native contacts|
  int n_p = 0;                            // native-identity (receptor atom, ligand atom) pairs
  int64_t counts[GD_EVAL_COUNTS] = {};    // as gd_evaluator_counts reports them
  const int *u_slot = nullptr;            // [n_u] device slot of each such ligand atom (interface atoms first)
  int n_if = 0;                           // the first n_if of them have an i-RMSD partner or native contacts
  // [n_u] ligand atom relative to the rotation centre in two limbs a coordinate
  // (x, y; z), then the paired reference atom relative to `origin` (x, y; z) in
  // 2^-51 A; w2 of u_z: bit 0: there is one; u_z.w >> 1: an i-RMSD partner of its own
  // (1), the same (2)
  const int4 *u_xy = nullptr, *u_z = nullptr;
  const longlong2 *u_qxy = nullptr;
  const long long *u_qz = nullptr;
  const D4 *u_ref = nullptr;              // [n_u] paired reference atom
  const D4 *u_iref = nullptr;             // [n_if] i-RMSD partner
  const Fix3 *u_iq = nullptr;             // [n_if] the same relative to `origin` in 2^-51 A
  bool fixed = false;                     // every coordinate is within the fixed-point range
  long long origin[3] = {0, 0, 0};        // the FP32 origin O rounded to whole Angstroms, in 2^-51 A
  const int *u_pbeg = nullptr;            // [n_if + 1] CSR offsets into p_rec
  const D4 *p_rec = nullptr;              // [n_p] receptor atoms whose contact with the ligand atom is native
  const float4 *p_rec32 = nullptr;        // [n_p] the same, FP32 relative to the origin O
  double thr5 = 0.0;
  void *block = nullptr;
  size_t bytes = 0;
};

namespace gd {
namespace {

struct EvalParams {
  ScoreParams p;  // ligand arrays, frames and the rotation centre
  const int *u_slot, *u_pbeg;
  const int4 *u_xy, *u_z;
  const longlong2 *u_qxy;
  const long long *u_qz;
  const Fix3 *u_iq;
  long long half;        // rotate()'s 2^28: from the arguments it costs no instructions (65,536 poses 1.070 -> 1.056 ms)
  long long ox, oy, oz;  // the evaluator's origin in 2^-51 A
  float fx, fy, fz;      // ... less the FP32 origin O
  bool fixed;
  const D4 *u_ref, *u_iref, *p_rec;
  const float4 *p_rec32;
  int n_u, n_if, n_ref, n_iref, n_native;
  double thr5;
  float extent;     // bounds |coordinate - O| of receptor and ligand atoms before the displacement
  const int *skip;  // nonzero: no work (a finished GA job); may be null
  gd_dock_metrics *out;
};

constexpr int kEvalWarps = 8;
constexpr int kEvalCtas = 3;    // resident per SM (registers)
// distance sums: a resolution of 2^-96 A (at the native pose the distances
// are rounding noise of some 1e-15 A), 2^31 A of room, single distances from
// 2^14 A on kept apart
constexpr int kDistBits = 96;
using DistSum = ExactSum<57>;

// The distance of ligand atom `slot` and (rx, ry, rz) as the reference forms
// it (exact transform, distance_to): out of line, few atoms come here.
__device__ __noinline__ double exact_distance(const ScoreParams &p, const gd_pose_frame &f, int pose, int slot,
                                              double rx, double ry, double rz) {
  double X, Y, Z;
  ligand_atom(p, f, pose, slot, X, Y, Z);
  return sqrt(exact_d2(X, Y, Z, rx, ry, rz));  // ligand atom first (src/evaluator.rs:96-100)
}

// The reference's contact decision (receptor atom first, src/evaluator.rs:150-152).
__device__ __noinline__ bool exact_contact(const ScoreParams &p, const gd_pose_frame &f, int pose, int slot, const D4 &a,
                                           double thr5) {
  double X, Y, Z;
  ligand_atom(p, f, pose, slot, X, Y, Z);
  return exact_d2(a.x, a.y, a.z, X, Y, Z) <= thr5;
}

// The length of (x, y, z) added to c 2^33 + r units of 2^-57 A, 2^-55 of it off
// at most (2^-51 from 64 A on); false below 1/4 A.  The squared length D (in
// 2^-68 A^2) differs from the square of its FP32 root s by R = D - s^2, some
// 2^-20 of it, formed exactly modulo 2^64; then
// sqrt(s^2 + R) = s + R / 2s - R^2 / 8s^3 + ... (the next term is 2^-60 of s),
// R / 2s as a multiple q of 2^20 units and an FP32 remainder.  Lengths with a
// coordinate from 64 A on are taken in 2^-45 A.  Conversions are of 32 bits:
// those of 64 run on the FP64 unit (seven of them an atom kept it 82 % busy and
// the kernel at 1.27 ms for 65,536 poses).
struct Length {
  unsigned s;  // 2^-24 A
  int q, tail;
  int far;     // all of them times 2^6
};
__device__ __forceinline__ bool fix_length(long long x, long long y, long long z, Length &o) {
  auto high = [](long long v) { return static_cast<int>((v + 0x80000000ll) >> 32); };
  auto size = [](int h) { return static_cast<unsigned>(h ^ (h >> 31)); };
  o.far = (size(high(x)) | size(high(y)) | size(high(z))) >= 64u << 19;
  if (o.far) {
    x = (x + 32) >> 6;
    y = (y + 32) >> 6;
    z = (z + 32) >> 6;
  }
  auto f32 = [](long long v) { return __int2float_rn(static_cast<int>((v + (1 << 26)) >> 27)); };  // in 2^-24 A
  const float gx = f32(x), gy = f32(y), gz = f32(z);
  const float d2 = __fmul_rn(__fmaf_rn(gz, gz, __fmaf_rn(gy, gy, __fmul_rn(gx, gx))), 0x1p-48f);
  if (!(d2 >= 0.0625f)) return false;
  float rs;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rs) : "f"(d2));
  o.s = __float2uint_rn(__fmul_rn(__fmul_rn(d2, rs), 16777216.0f));
  const int hx = high(x), hy = high(y), hz = high(z), lx = static_cast<int>(x), ly = static_cast<int>(y),
            lz = static_cast<int>(z);
  const long long hl = static_cast<long long>(hx) * lx + static_cast<long long>(hy) * ly + static_cast<long long>(hz) * lz;
  const unsigned long long hh = static_cast<long long>(hx) * hx + static_cast<long long>(hy) * hy + static_cast<long long>(hz) * hz;
  const unsigned long long ll = static_cast<unsigned long long>(static_cast<long long>(lx) * lx) +
                                static_cast<unsigned long long>(static_cast<long long>(ly) * ly) +
                                static_cast<unsigned long long>(static_cast<long long>(lz) * lz);
  const unsigned long long D = static_cast<unsigned long long>(hl >> 1) + (ll >> 34) + (hh << 30);
  // R to 2^-64 of d2: 46 bits in two exact FP32 parts
  const int up = (__float_as_int(d2) >> 23) - 127 + 4;
  const long long R = static_cast<long long>(D - ((static_cast<unsigned long long>(o.s) * o.s) << 20)) >> up;
  const float rh = __fmul_rn(__int2float_rn(static_cast<int>(R >> 22)), 4194304.0f);
  const float rl = __int2float_rn(static_cast<int>(R) & 0x3fffff);
  const float w = __fmul_rn(__fmul_rn(rs, 0x1p-12f), __int_as_float((127 + up) << 23));
  const float s12 = __fmul_rn(__fmul_rn(__uint2float_rn(o.s), 0x1p-12f), __int_as_float((127 - up) << 23));
  o.q = __float2int_rn(__fmul_rn(__fmul_rn(rh, w), 0x1p-20f));
  const float qf = __fmul_rn(__int2float_rn(o.q), 0x1p20f);
  const float rem = __fadd_rn(__fmaf_rn(-qf, s12, rh), rl);
  o.tail = __float2int_rn(__fmaf_rn(rem, w, -__fmul_rn(__fmul_rn(qf, qf), __fmul_rn(rs, 0x1p-58f))));
  return true;
}

struct FarSum { __int128 v; double nf; };

// A thread's distance sums: fix_length()'s in registers, those formed in FP64
// (few, or all of a pose out of range) in shared memory, touched when there is
// one.
struct PoseSum {
  unsigned long long c = 0;
  long long r = 0;
  __device__ __forceinline__ void add(const Length &d) {
    const int unit = d.far ? 64 : 1;
    c += static_cast<unsigned long long>(d.s) * static_cast<unsigned>(unit);
    r += static_cast<long long>(d.q) * (unit << 20);
    r += static_cast<long long>(d.tail) * unit;
  }
  __device__ __forceinline__ DistSum close(const FarSum &far, bool used) const {
    DistSum d;
    if (used) {
      d.v = far.v;
      d.nf = far.nf;
    }
    d.v += ((static_cast<__int128>(c) << 33) + r) << (kDistBits - 57);
    return d;
  }
};
// A finished pose, until its warp has 32.
struct Held {
  __int128 l, i;
  double nf_l, nf_i;
  int common, pose;
};

// What bounds it: instruction issue and the integer multiply-add unit.  FP64
// issues once in 64 cycles, so the FP64 form (12 operations for an atom's
// difference from its partner, 8 for square and root) kept that pipe 85 % busy;
// in fixed point an atom is some 230 integer and FP32 instructions on units
// thirty times as fast, and the result is closer.  Three CTAs an SM measured
// best (two: 3 % slower, four: spills, 5 %).  WPP warps per pose: one where the
// poses fill the GPU, else the whole CTA (150 poses of one warp each kept 38 of
// the 152 SMs waiting).
// 65,536 poses of 2,538 x 1,280 atoms (the whole call, host frames and copies
// included): 10.8 ms in the reference's operation order, 4.18 as FP64
// multiply-add chains (the kernel 3.53), 1.69 in fixed point (0.99).
template <int WPP>
__global__ void __launch_bounds__(kEvalWarps * 32, kEvalCtas) k_dockq(const EvalParams e) {
  if (e.skip && *e.skip) return;
  __shared__ gd_pose_frame s_f[kEvalWarps / WPP];
  __shared__ Limbs s_m[kEvalWarps][9];
  __shared__ long long s_t[kEvalWarps][3];
  __shared__ __int128 s_sum[kEvalWarps][2];
  __shared__ double s_nf[kEvalWarps][2];
  __shared__ int s_common[kEvalWarps];
  __shared__ Held s_held[WPP == 1 ? kEvalWarps * 32 : 32];
  __shared__ FarSum s_far[kEvalWarps * 32][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int step = gridDim.x * (kEvalWarps / WPP);
  const int t0 = WPP == 1 ? lane : static_cast<int>(threadIdx.x);
  gd_pose_frame &f = s_f[WPP == 1 ? warp : 0];
  // a warp keeps the poses' sums until it has 32 of them: the divisions and
  // roots of the metrics then run on all lanes
  Held *my = s_held + (WPP == 1 ? warp * 32 : 0);
  int held = 0;
  auto finish = [&]() {
    __syncwarp();
    if (lane < held) {
      // src/evaluator.rs:68-84, without contraction into fused multiply-adds
      const Held &h = my[lane];
      DistSum l, i;
      l.v = h.l;
      l.nf = h.nf_l;
      i.v = h.i;
      i.nf = h.nf_i;
      const double sl = l.value(kDistBits), si = i.value(kDistBits);
      const double rmsd = e.n_ref ? __dsqrt_rn(__ddiv_rn(sl, static_cast<double>(e.n_ref))) : 0.0;
      const double irmsd = e.n_iref ? __dsqrt_rn(__ddiv_rn(si, static_cast<double>(e.n_iref))) : 0.0;
      const double fnat = e.n_native ? __ddiv_rn(static_cast<double>(h.common), static_cast<double>(e.n_native)) : 0.0;
      const double a = __ddiv_rn(irmsd, 1.5), b = __ddiv_rn(rmsd, 8.5);
      const double is = __ddiv_rn(1.0, __dadd_rn(1.0, __dmul_rn(a, a)));
      const double ls = __ddiv_rn(1.0, __dadd_rn(1.0, __dmul_rn(b, b)));
      const double dockq = __ddiv_rn(__dadd_rn(__dadd_rn(fnat, is), ls), 3.0);
      e.out[h.pose] = gd_dock_metrics{rmsd, irmsd, fnat, dockq};
    }
    __syncwarp();
    held = 0;
  };
  for (int pose = blockIdx.x * (kEvalWarps / WPP) + (WPP == 1 ? warp : 0); pose < e.p.n_poses; pose += step) {
    if (WPP == 1) __syncwarp();
    else __syncthreads();
    if (t0 < 16) reinterpret_cast<double *>(&f)[t0] = reinterpret_cast<const double *>(e.p.frames + pose)[t0];
    if (WPP == 1) __syncwarp();
    else __syncthreads();
    // the rotation (src/structure.rs:80-131) and the centre + displacement in
    // fixed point, an entry a lane, as a sum of two doubles: a product and what
    // its rounding drops, the centre and the displacement (the error of either
    // one's rounded value is the same for every atom).  fix: all of them are in
    // range, by their high words.
    bool ok = true;
    if (lane < 12) {
      const bool turn = lane < 9;
      const double a = lane == 0 ? f.ca : lane == 1 ? f.m01 : lane == 2 ? f.m02 : lane == 3 ? f.sa : lane == 4 ? f.m11
                       : lane == 5 ? f.m12 : lane == 6 ? -f.sb : turn ? f.cb : lane == 9 ? e.p.cx : lane == 10 ? e.p.cy : e.p.cz;
      const double b = lane == 0 || lane == 3 ? f.cb : lane == 7 ? f.sg : lane == 8 ? f.cg : 1.0;
      const double m = __dmul_rn(a, b), rest = __fma_rn(a, b, -m);
      const double d = turn ? rest : lane == 9 ? f.dx : lane == 10 ? f.dy : f.dz, one = turn ? 0x1p59 : 0x1p51;
      const int most = __double2hiint(turn ? 1.5 : 4000.0);
      auto below = [&](double v) { return (__double2hiint(v) & 0x7fffffff) < most; };
      ok = below(m) && below(d) && below(m + d);
      const long long v = ok ? __double2ll_rn(m * one) + __double2ll_rn(d * one) : 0;
      if (turn) {
        s_m[warp][lane] = limbs(v);
      } else {
        const long long t = v - (lane == 9 ? e.ox : lane == 10 ? e.oy : e.oz);
        ok = ok && llabs(t) < static_cast<long long>(kFixFar * 0x1p51);
        s_t[warp][lane - 9] = t;
      }
    }
    const bool fix = __all_sync(kFull, ok) && e.fixed;
    __syncwarp();
    Limbs m[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) m[k] = s_m[warp][k];
    const long long tx = s_t[warp][0], ty = s_t[warp][1], tz = s_t[warp][2];
    // the FP32 guard band of the contact test, as for the contact lists
    // (M bounds the coordinates; twice it covers the sum that forms them)
    const float M = 2.0f * (e.extent + fmaxf(fabsf(static_cast<float>(f.dx)),
                                             fmaxf(fabsf(static_cast<float>(f.dy)), fabsf(static_cast<float>(f.dz)))));
    const float guard = 4.0f * (17.33f * (2.0f * M + 5.0f) + 100.0f) * 0x1p-24f + 1e-6f;
    const bool band_ok = guard < 1.0f && fix;
    PoseSum sl, si;
    int common = 0;
    FarSum *far = s_far[threadIdx.x];
    bool used = false;
    auto add_far = [&](double d, bool to_l, bool to_i) {
      if (!used) far[0] = far[1] = FarSum{0, 0.0};
      used = true;
      DistSum v;
      v.add(d, kDistBits);
      for (int k = 0; k < 2; ++k)
        if (k == 0 ? to_l : to_i) {
          far[k].v += v.v;
          far[k].nf += v.nf;
        }
    };
#pragma unroll 1
    for (int u = t0; u < e.n_u; u += 32 * WPP) {
      const int4 xy = e.u_xy[u], z = e.u_z[u];
      const long long px = rotate(m[0], m[1], m[2], xy, z, e.half) + tx, py = rotate(m[3], m[4], m[5], xy, z, e.half) + ty,
                      pz = rotate(m[6], m[7], m[8], xy, z, e.half) + tz;
      auto slot = [&]() {
        const int sl = e.u_slot[u];
        return GD_DCHECK(e.p.err, sl >= 0 && sl < e.p.nl, 40) ? sl : 0;
      };
      const int iw = z.w >> 1;
      if (z.w & 1) {
        const longlong2 q = e.u_qxy[u];
        Length d;
        if (fix && fix_length(px - q.x, py - q.y, pz - e.u_qz[u], d)) {
          sl.add(d);
          if (iw == 2) si.add(d);
        } else {
          const D4 a = e.u_ref[u];
          add_far(exact_distance(e.p, f, pose, slot(), a.x, a.y, a.z), true, iw == 2);
        }
      }
      if (u < e.n_if) {
        if (iw == 1) {
          const Fix3 q = e.u_iq[u];
          Length d;
          if (fix && fix_length(px - q.x, py - q.y, pz - q.z, d)) {
            si.add(d);
          } else {
            const D4 a = e.u_iref[u];
            add_far(exact_distance(e.p, f, pose, slot(), a.x, a.y, a.z), false, true);
          }
        }
        int k = e.u_pbeg[u];
        const int k1 = e.u_pbeg[u + 1];
        if (k < k1) {
          auto f32 = [](long long v, float o) {
            const int h = static_cast<int>((v + 0x80000000ll) >> 32);
            return __fmaf_rn(__int2float_rn(static_cast<int>(v)), 0x1p-51f, __fmaf_rn(__int2float_rn(h), 0x1p-19f, o));
          };
          const float lx = f32(px, e.fx), ly = f32(py, e.fy), lz = f32(pz, e.fz);
          for (; k < k1; ++k) {
            const float t = d2f(__ldg(&e.p_rec32[k]), lx, ly, lz) - 25.0f;
            bool hit = t < 0.0f;
            if (!(band_ok && fabsf(t) > guard)) hit = exact_contact(e.p, f, pose, slot(), e.p_rec[k], e.thr5);
            common += hit;
          }
        }
      }
    }
    DistSum dl = sl.close(far[0], used), di = si.close(far[1], used);
    dl.warp_total();
    di.warp_total();
    common = __reduce_add_sync(kFull, common);
    if (WPP > 1) {
      if (lane == 0) {
        s_sum[warp][0] = dl.v;
        s_sum[warp][1] = di.v;
        s_nf[warp][0] = dl.nf;
        s_nf[warp][1] = di.nf;
        s_common[warp] = common;
      }
      __syncthreads();
      if (warp == 0) {
        for (int w = 1; w < WPP; ++w) {
          dl.v += s_sum[w][0];
          di.v += s_sum[w][1];
          dl.nf += s_nf[w][0];
          di.nf += s_nf[w][1];
          common += s_common[w];
        }
      }
    }
    if (WPP == 1 || warp == 0) {
      if (lane == 0) {
        my[held] = Held{dl.v, di.v, dl.nf, di.nf, common, pose};
      }
      if (++held == 32) finish();
    }
  }
  if (WPP == 1 || warp == 0) finish();
}

double host_dist(double ax, double ay, double az, double bx, double by, double bz) {
  const double dx = ax - bx, dy = ay - by, dz = az - bz;
  return std::sqrt(dx * dx + dy * dy + dz * dz);
}

}  // namespace

gd_complex *evaluator_complex(const gd_evaluator *ev) { return ev->cx; }

gd_status launch_dockq(gd_evaluator *ev, const gd_pose_frame *d_frames, int n, gd_dock_metrics *d_out,
                       const int *skip, cudaStream_t stream) {
  if (n == 0) return GD_OK;
  EvalParams ep{};
  ep.p = make_params(ev->cx, d_frames, nullptr, n, nullptr, 0.0);
  ep.u_slot = ev->u_slot;
  ep.u_pbeg = ev->u_pbeg;
  ep.u_xy = ev->u_xy;
  ep.u_z = ev->u_z;
  ep.u_qxy = ev->u_qxy;
  ep.u_qz = ev->u_qz;
  ep.u_iq = ev->u_iq;
  ep.half = 1 << 28;
  ep.ox = ev->origin[0];
  ep.oy = ev->origin[1];
  ep.oz = ev->origin[2];
  ep.fx = static_cast<float>(std::ldexp(static_cast<double>(ev->origin[0]), -51) - ev->cx->ox);
  ep.fy = static_cast<float>(std::ldexp(static_cast<double>(ev->origin[1]), -51) - ev->cx->oy);
  ep.fz = static_cast<float>(std::ldexp(static_cast<double>(ev->origin[2]), -51) - ev->cx->oz);
  ep.fixed = ev->fixed;
  ep.u_ref = ev->u_ref;
  ep.u_iref = ev->u_iref;
  ep.p_rec = ev->p_rec;
  ep.p_rec32 = ev->p_rec32;
  ep.n_u = ev->n_u;
  ep.n_if = ev->n_if;
  ep.n_ref = ev->n_ref;
  ep.n_iref = ev->n_iref;
  ep.n_native = ev->n_native;
  ep.thr5 = ev->thr5;
  const gd_complex *cx = ev->cx;
  const double m = std::max(cx->rec_extent, cx->lig_radius + std::max({std::fabs(cx->cx - cx->ox), std::fabs(cx->cy - cx->oy),
                                                                      std::fabs(cx->cz - cx->oz)})) + 1.0;
  ep.extent = static_cast<float>(m * (1.0 + 1e-6));
  ep.skip = skip;
  ep.out = d_out;
  // one warp per pose when the poses give two of three resident warps one, else
  // a CTA per pose (2,538 x 1,280 atoms, the call with its host frames: 1,500
  // poses 169 us a warp each, 154 a CTA each, 2,500 poses 248 and 253, 5,000
  // poses 249 and 313; 841 x 170 atoms, 1,000 poses 83 and 93)
  const int warps = kEvalCtas * kEvalWarps * ev->ctx->sm_count;
  if (n >= warps * 2 / 3)
    k_dockq<1><<<std::min((n + kEvalWarps - 1) / kEvalWarps, warps / kEvalWarps), kEvalWarps * 32, 0, stream>>>(ep);
  else
    k_dockq<kEvalWarps><<<n, kEvalWarps * 32, 0, stream>>>(ep);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GD_OK : cuda_fail(ev->ctx, e, "evaluator launch");
}

}  // namespace gd

using namespace gd;

extern "C" {

gd_status gd_evaluator_create(gd_complex *cx, const gd_atoms *reference, const uint32_t *rec_names,
                              const uint32_t *lig_names, const uint32_t *ref_names, gd_evaluator **out) {
  gd::NvtxRange nvtx_range("gd_evaluator_create");
  if (!cx || !reference || !out) return GD_ERR_INVALID_ARG;
  gd_context *ctx = cx->ctx;
  *out = nullptr;
  const int nr = static_cast<int>(cx->h_rx.size()), nl = static_cast<int>(cx->h_lx.size()), nf = reference->n;
  if (nf < 0 || (nf > 0 && (!reference->x || !reference->y || !reference->z || !reference->resseq ||
                            !reference->chain || !ref_names)) ||
      (nr > 0 && !rec_names) || (nl > 0 && !lig_names))
    return fail(ctx, GD_ERR_INVALID_ARG, "bad reference or atom names");
  cudaSetDevice(ctx->device);
  // interface residues (src/evaluator.rs:170-186)
  std::set<int16_t> rec_if, ref_if;
  for (int a = 0; a < nr; ++a)
    for (int b = 0; b < nf; ++b)
      if (host_dist(cx->h_rx[a], cx->h_ry[a], cx->h_rz[a], reference->x[b], reference->y[b], reference->z[b]) <=
          5.0) {
        rec_if.insert(cx->h_rres[a]);
        ref_if.insert(reference->resseq[b]);
      }
  std::vector<int> rec_i, ref_i, lig_i;  // interface atoms, in order
  for (int a = 0; a < nr; ++a)
    if (rec_if.count(cx->h_rres[a])) rec_i.push_back(a);
  for (int b = 0; b < nf; ++b)
    if (ref_if.count(reference->resseq[b])) ref_i.push_back(b);
  for (int j = 0; j < nl; ++j)
    if (ref_if.count(cx->h_lres[j])) lig_i.push_back(j);
  // native contacts: identities (chain, residue, name) of both atoms
  using Id = std::tuple<uint8_t, int16_t, uint32_t, uint8_t, int16_t, uint32_t>;
  std::set<Id> native_set;
  int n_native = 0;
  for (int a : rec_i)
    for (int b : ref_i)
      if (host_dist(cx->h_rx[a], cx->h_ry[a], cx->h_rz[a], reference->x[b], reference->y[b], reference->z[b]) <=
          5.0) {
        native_set.insert(Id{cx->h_rchain[a], cx->h_rres[a], rec_names[a], reference->chain[b],
                             reference->resseq[b], ref_names[b]});
        ++n_native;
      }
  // per ligand atom (in device slot order): its L-RMSD partner (the
  // reference atom of the same index: zip truncates at the shorter), its
  // i-RMSD partner (same rank among the interface atoms of both), and the
  // receptor interface atoms whose contact with it has a native identity
  std::vector<D4> l_ref(nl, D4{0, 0, 0, 0}), l_iref(nl, D4{0, 0, 0, 0});
  std::vector<std::vector<int>> l_rec(nl);
  for (int k = 0; k < std::min(nl, nf); ++k) l_ref[k] = D4{reference->x[k], reference->y[k], reference->z[k], 1.0};
  for (size_t k = 0; k < std::min(lig_i.size(), ref_i.size()); ++k) {
    const int b = ref_i[k];
    l_iref[lig_i[k]] = D4{reference->x[b], reference->y[b], reference->z[b], 1.0};
  }
  int n_p = 0;
  for (int a : rec_i)
    for (int j : lig_i)
      if (native_set.count(Id{cx->h_rchain[a], cx->h_rres[a], rec_names[a], cx->h_lchain[j], cx->h_lres[j],
                              lig_names[j]})) {
        l_rec[j].push_back(a);
        ++n_p;
      }
  // ligand atoms the metrics read: the interface ones (i-RMSD pairing or
  // contacts) first, so that the warps' branches for them stay uniform, then
  // the rest; each group by device slot
  std::vector<int> order;
  for (int j = 0; j < nl; ++j)
    if (l_ref[j].w != 0.0 || l_iref[j].w != 0.0 || !l_rec[j].empty()) order.push_back(j);
  auto group = [&](int j) { return (l_iref[j].w != 0.0 || !l_rec[j].empty()) ? 0 : 1; };
  std::sort(order.begin(), order.end(), [&](int x, int y) {
    return group(x) != group(y) ? group(x) < group(y) : cx->h_lig_slot[x] < cx->h_lig_slot[y];
  });
  const int nu = static_cast<int>(order.size());
  int n_if = 0;
  while (n_if < nu && group(order[n_if]) == 0) ++n_if;
  std::vector<int> u_slot(nu), u_pbeg(n_if + 1, 0);
  std::vector<D4> u_ref(nu), u_iref(n_if), p_rec;
  std::vector<int4> u_xy(nu, make_int4(0, 0, 0, 0)), u_z(nu, make_int4(0, 0, 0, 0));
  std::vector<longlong2> u_qxy(nu, longlong2{0, 0});
  std::vector<long long> u_qz(nu, 0);
  std::vector<Fix3> u_iq(n_if, Fix3{0, 0, 0, 0});
  // the fixed-point images, as long as every coordinate is in range
  bool fixed = std::max({std::fabs(cx->ox), std::fabs(cx->oy), std::fabs(cx->oz)}) < 3000.0;
  const double whole[3] = {fixed ? std::nearbyint(cx->ox) : 0.0, fixed ? std::nearbyint(cx->oy) : 0.0,
                           fixed ? std::nearbyint(cx->oz) : 0.0};
  long long origin[3];
  for (int k = 0; k < 3; ++k) origin[k] = fix_int(whole[k], 0x1p51);
  auto fix_ref = [&](const D4 &v) {
    if (!(std::fabs(v.x) < 4000.0 && std::fabs(v.y) < 4000.0 && std::fabs(v.z) < 4000.0)) {
      fixed = false;
      return Fix3{0, 0, 0, 0};
    }
    const Fix3 q{fix_int(v.x, 0x1p51) - origin[0], fix_int(v.y, 0x1p51) - origin[1],
                 fix_int(v.z, 0x1p51) - origin[2], 0};
    const long long lim = fix_int(kFixFar, 0x1p51);
    fixed = fixed && std::llabs(q.x) < lim && std::llabs(q.y) < lim && std::llabs(q.z) < lim;
    return q;
  };
  std::vector<float4> p_rec32;
  p_rec.reserve(n_p);
  p_rec32.reserve(n_p);
  for (int u = 0; u < nu; ++u) {
    const int j = order[u];
    u_slot[u] = cx->h_lig_slot[j];
    const double x0[3] = {cx->h_lx[j] - cx->cx, cx->h_ly[j] - cx->cy, cx->h_lz[j] - cx->cz};
    if (std::fabs(x0[0]) < kFixAtom && std::fabs(x0[1]) < kFixAtom && std::fabs(x0[2]) < kFixAtom) {
      const Limbs x = limbs(fix_int(x0[0], 0x1p50)), y = limbs(fix_int(x0[1], 0x1p50)),
                  z = limbs(fix_int(x0[2], 0x1p50));
      u_xy[u] = make_int4(x.h, x.l, y.h, y.l);
      u_z[u] = make_int4(z.h, z.l, 0, 0);
    } else {
      fixed = false;
    }
    u_ref[u] = l_ref[j];
    if (l_ref[j].w != 0.0) {
      const Fix3 q = fix_ref(l_ref[j]);
      u_qxy[u] = longlong2{q.x, q.y};
      u_qz[u] = q.z;
      u_z[u].w = 1;
    }
    if (u >= n_if) continue;
    u_iref[u] = l_iref[j];
    if (l_iref[j].w != 0.0) {
      u_iq[u] = fix_ref(l_iref[j]);
      const bool same = l_ref[j].w != 0.0 && l_ref[j].x == l_iref[j].x && l_ref[j].y == l_iref[j].y && l_ref[j].z == l_iref[j].z;
      u_z[u].w |= same ? 4 : 2;
    }
    for (int a : l_rec[j]) {
      p_rec.push_back(D4{cx->h_rx[a], cx->h_ry[a], cx->h_rz[a], 0.0});
      p_rec32.push_back(make_float4(static_cast<float>(cx->h_rx[a] - cx->ox), static_cast<float>(cx->h_ry[a] - cx->oy),
                                    static_cast<float>(cx->h_rz[a] - cx->oz), 0.0f));
    }
    u_pbeg[u + 1] = static_cast<int>(p_rec.size());
  }
  gd_evaluator *ev = new gd_evaluator();
  ev->cx = cx;
  ev->ctx = ctx;
  ev->n_u = nu;
  ev->n_if = n_if;
  ev->n_ref = nf;
  ev->n_iref = static_cast<int>(ref_i.size());
  ev->n_native = n_native;
  ev->n_p = n_p;
  ev->fixed = fixed;
  std::copy(origin, origin + 3, ev->origin);
  ev->thr5 = make_thresholds(5.0).contact_le;
  const int64_t cnt[GD_EVAL_COUNTS] = {static_cast<int64_t>(rec_if.size()), static_cast<int64_t>(ref_if.size()),
                                       n_native, nu, std::min(nl, nf),
                                       static_cast<int64_t>(std::min(lig_i.size(), ref_i.size())), n_p};
  std::copy(cnt, cnt + GD_EVAL_COUNTS, ev->counts);
  auto al = [](size_t b) { return (std::max<size_t>(b, 1) + 255) / 256 * 256; };
  const size_t b_slot = al(sizeof(int) * nu), b_beg = al(sizeof(int) * (n_if + 1)), b_ref = al(sizeof(D4) * nu),
               b_iref = al(sizeof(D4) * n_if), b_x = al(sizeof(int4) * nu), b_qz = al(sizeof(long long) * nu), b_prec = al(sizeof(D4) * p_rec.size()),
               b_prec32 = al(sizeof(float4) * p_rec32.size());
  ev->bytes = b_slot + b_beg + b_ref + 2 * b_iref + 3 * b_x + b_qz + b_prec + b_prec32;
  gd_status s = dev_alloc(ctx, ev->bytes, &ev->block);
  if (s != GD_OK) {
    delete ev;
    return s;
  }
  std::vector<char> h(ev->bytes, 0);
  size_t o = 0;
  auto put = [&](const void *src, size_t n, size_t b) {
    if (n) std::memcpy(h.data() + o, src, n);
    char *d = static_cast<char *>(ev->block) + o;
    o += b;
    return d;
  };
  ev->u_slot = reinterpret_cast<const int *>(put(u_slot.data(), sizeof(int) * nu, b_slot));
  ev->u_pbeg = reinterpret_cast<const int *>(put(u_pbeg.data(), sizeof(int) * (n_if + 1), b_beg));
  ev->u_xy = reinterpret_cast<const int4 *>(put(u_xy.data(), sizeof(int4) * nu, b_x));
  ev->u_z = reinterpret_cast<const int4 *>(put(u_z.data(), sizeof(int4) * nu, b_x));
  ev->u_qxy = reinterpret_cast<const longlong2 *>(put(u_qxy.data(), sizeof(longlong2) * nu, b_x));
  ev->u_qz = reinterpret_cast<const long long *>(put(u_qz.data(), sizeof(long long) * nu, b_qz));
  ev->u_iq = reinterpret_cast<const Fix3 *>(put(u_iq.data(), sizeof(Fix3) * n_if, b_iref));
  ev->u_ref = reinterpret_cast<const D4 *>(put(u_ref.data(), sizeof(D4) * nu, b_ref));
  ev->u_iref = reinterpret_cast<const D4 *>(put(u_iref.data(), sizeof(D4) * n_if, b_iref));
  ev->p_rec = reinterpret_cast<const D4 *>(put(p_rec.data(), sizeof(D4) * p_rec.size(), b_prec));
  ev->p_rec32 = reinterpret_cast<const float4 *>(put(p_rec32.data(), sizeof(float4) * p_rec32.size(), b_prec32));
  const cudaError_t e = cudaMemcpy(ev->block, h.data(), ev->bytes, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    dev_free(ctx, ev->block, ev->bytes);
    delete ev;
    return cuda_fail(ctx, e, "evaluator upload");
  }
  *out = ev;
  return GD_OK;
}

gd_status gd_evaluator_counts(const gd_evaluator *ev, int64_t *counts) {
  if (!ev || !counts) return GD_ERR_INVALID_ARG;
  std::copy(ev->counts, ev->counts + GD_EVAL_COUNTS, counts);
  return GD_OK;
}

gd_status gd_evaluator_destroy(gd_evaluator *ev) {
  if (!ev) return GD_ERR_INVALID_ARG;
  gd_context *ctx = ev->ctx;
  cudaSetDevice(ctx->device);
  if (ev->block) dev_free(ctx, ev->block, ev->bytes);
  delete ev;
  return GD_OK;
}

gd_status gd_evaluate_frames_device(gd_evaluator *ev, const gd_pose_frame *d_frames, int32_t n,
                                    gd_dock_metrics *d_out, void *stream) {
  if (!ev) return GD_ERR_INVALID_ARG;
  gd_context *ctx = ev->ctx;
  if (n < 0 || (n > 0 && (!d_frames || !d_out))) return fail(ctx, GD_ERR_INVALID_ARG, "bad frames/out");
  cudaSetDevice(ctx->device);
  return launch_dockq(ev, d_frames, n, d_out, nullptr, stream ? static_cast<cudaStream_t>(stream) : ctx->stream);
}

gd_status gd_evaluate_poses(gd_evaluator *ev, const double *genes, int32_t n, gd_dock_metrics *out) {
  gd::NvtxRange nvtx_range("gd_evaluate_poses");
  if (!ev) return GD_ERR_INVALID_ARG;
  gd_context *ctx = ev->ctx;
  if (n < 0 || (n > 0 && (!genes || !out))) return fail(ctx, GD_ERR_INVALID_ARG, "bad genes/out");
  if (n == 0) return GD_OK;
  cudaSetDevice(ctx->device);
  const size_t fb = sizeof(gd_pose_frame) * n, ob = sizeof(gd_dock_metrics) * n;
  const size_t fb_al = (fb + 255) / 256 * 256;
  const bool staged = fb_al + ob <= kStageMax;
  const ScratchUse use(ctx);
  gd_status s = ensure_scratch(ctx, fb_al + ob, staged ? fb_al + ob : 0);
  if (s != GD_OK) return s;
  gd_pose_frame *d_frames = static_cast<gd_pose_frame *>(ctx->d_scratch);
  gd_dock_metrics *d_out = reinterpret_cast<gd_dock_metrics *>(static_cast<char *>(ctx->d_scratch) + fb_al);
  std::vector<gd_pose_frame> pageable(staged ? 0 : n);
  gd_pose_frame *frames = staged ? static_cast<gd_pose_frame *>(ctx->h_pinned) : pageable.data();
  void *res = staged ? static_cast<char *>(ctx->h_pinned) + fb_al : static_cast<void *>(out);
  gd_make_frames(genes, n, frames);
  cudaStream_t st = ctx->stream;
  const bool direct = staged && n <= kDirectPoses;  // frames and metrics in the staging buffer itself
  cudaError_t e = direct ? cudaSuccess : cudaMemcpyAsync(d_frames, frames, fb, cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "evaluator frames upload");
  s = gd_evaluate_frames_device(ev, direct ? frames : d_frames, n, direct ? static_cast<gd_dock_metrics *>(res) : d_out, st);
  if (s == GD_OK && !direct) {
    e = cudaMemcpyAsync(res, d_out, ob, cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) s = cuda_fail(ctx, e, "evaluator");
  }
  if (s != GD_OK) {
    cudaStreamSynchronize(st);
    return s;
  }
  s = finish_stream(ctx, st, "evaluator");
  if (s == GD_OK && staged) copy_out(out, res, ob);
  return s;
}

}  // extern "C"
