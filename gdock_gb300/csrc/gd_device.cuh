// Device helpers shared by the scoring kernels: bulk-copy/mbarrier
// primitives (inline PTX), the exact pose transform, exact squared distance,
// warp sums, and the per-pose AIR/record epilogue.
#pragma once

#include "gd_internal.cuh"

namespace gd {

constexpr unsigned kFull = 0xffffffffu;

static __device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
static __device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
static __device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
static __device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
// 1-D bulk copy global -> shared (the TMA engine), completing on an mbarrier.
static __device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
static __device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
static __device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait on an mbarrier phase: false after kWaitLimitNs of wall time
// (or kSpinLimit polls), so that a copy that never lands ends the kernel
// with an error instead of a hang.
static __device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  for (uint32_t i = 1; i < kSpinLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 0 && global_ns() - t0 > kWaitLimitNs) return false;
  }
  return false;
}

static __device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Rigid transform of one ligand atom with the reference's operation order
// (src/structure.rs:83-115, then displace :119-131); explicit _rn intrinsics
// keep the compiler from fusing multiply-adds, so the result is bit-identical
// to the host's double arithmetic.
static __device__ __forceinline__ void transform_atom(const gd_pose_frame &f, double cx, double cy, double cz,
                                               double xo, double yo, double zo, double &X, double &Y,
                                               double &Z) {
  const double x = __dsub_rn(xo, cx), y = __dsub_rn(yo, cy), z = __dsub_rn(zo, cz);
  const double nx = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(x, f.ca), f.cb), __dmul_rn(y, f.m01)),
                              __dmul_rn(z, f.m02));
  const double ny = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(x, f.sa), f.cb), __dmul_rn(y, f.m11)),
                              __dmul_rn(z, f.m12));
  const double nz = __dadd_rn(__dadd_rn(__dmul_rn(-x, f.sb), __dmul_rn(__dmul_rn(y, f.cb), f.sg)),
                              __dmul_rn(__dmul_rn(z, f.cb), f.cg));
  X = __dadd_rn(__dadd_rn(nx, cx), f.dx);
  Y = __dadd_rn(__dadd_rn(ny, cy), f.dy);
  Z = __dadd_rn(__dadd_rn(nz, cz), f.dz);
}

// Exact ligand coordinates of atom j of the current pose.
static __device__ __forceinline__ void ligand_atom(const ScoreParams &p, const gd_pose_frame &f, int pose, int j,
                                            double &X, double &Y, double &Z) {
  if (p.models) {
    const double *m = p.models + (static_cast<size_t>(pose) * p.nl + p.lig_perm[j]) * 3;  // models: original order
    X = m[0];
    Y = m[1];
    Z = m[2];
  } else {
    transform_atom(f, p.cx, p.cy, p.cz, p.lig_x[j], p.lig_y[j], p.lig_z[j], X, Y, Z);
  }
}

// structure::distance squared, (dx*dx + dy*dy) + dz*dz (src/structure.rs:312-317)
static __device__ __forceinline__ double exact_d2(double ax, double ay, double az, double bx, double by, double bz) {
  const double dx = __dsub_rn(ax, bx), dy = __dsub_rn(ay, by), dz = __dsub_rn(az, bz);
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// Ligand coordinates relative to the FP32 origin O, in FP64, as the FP32 images
// are rounded from where fixed point does not reach, and for the slots' spheres:
// one chain of multiply-adds on the precomputed offset from the rotation centre,
// 9 FP64 operations in place of the 31 of the reference's order, from which it
// differs by some 1e-15 A (decisions inside the guard bands take the exact
// coordinates).
static __device__ __forceinline__ void relative_atom(const ScoreParams &p, const gd_pose_frame &f, const D4 &r, double &x,
                                                     double &y, double &z) {
  const double tx = (p.cx + f.dx) - p.ox, ty = (p.cy + f.dy) - p.oy, tz = (p.cz + f.dz) - p.oz;
  x = __fma_rn(f.ca * f.cb, r.x, __fma_rn(f.m01, r.y, __fma_rn(f.m02, r.z, tx)));
  y = __fma_rn(f.sa * f.cb, r.x, __fma_rn(f.m11, r.y, __fma_rn(f.m12, r.z, ty)));
  z = __fma_rn(-f.sb, r.x, __fma_rn(f.cb * f.sg, r.y, __fma_rn(f.cb * f.cg, r.z, tz)));
}
// One coordinate of the rotated atom: nine 32 x 32 -> 64 multiply-adds of
// three products, the low limbs' dropped.  Those are of either sign and the sum
// is rounded, so that the error, five quarters of a unit of 2^-51 A at most, is as
// often up as down and averages out over a pose's atoms (limbs from 0 up and a
// sum rounded down put every atom 5e-16 A to one side on average).  An FP64 chain
// of multiply-adds errs by ten times as much at 60 A.  half: what rounds the sum.
static __device__ __forceinline__ long long rotate(const Limbs &a, const Limbs &b, const Limbs &c, const int4 &xy, const int4 &z, long long half = 1 << 28) {
  long long hi = static_cast<long long>(a.h) * xy.x, mid = static_cast<long long>(a.h) * xy.y + half;
  hi += static_cast<long long>(b.h) * xy.z;
  mid += static_cast<long long>(a.l) * xy.x;
  hi += static_cast<long long>(c.h) * z.x;
  mid += static_cast<long long>(b.h) * xy.w;
  mid += static_cast<long long>(b.l) * xy.z;
  mid += static_cast<long long>(c.h) * z.y;
  mid += static_cast<long long>(c.l) * z.x;
  return hi + (mid >> 29);
}

// v 2^-51 as a float (v below 2^63): off by the rounding of the sum and, the low
// part having been rounded to 24 bits first, by another 2^-36 A at most.
static __device__ __forceinline__ float fix_float(long long v) {
  const float hi = __int2float_rn(static_cast<int>(v >> 40)), lo = __uint2float_rn(static_cast<unsigned>(v >> 8));
  return __fmul_rn(__fmaf_rn(lo, 0x1p-32f, hi), 0x1p-11f);
}

// The squared length of d (2^-51 A, below 16 A) in 2^-56 A^2: exact squares,
// truncated.
static __device__ __forceinline__ unsigned long long fix_d2(const long long *d) {
  long long H = 0, M = 0;
  unsigned lo = 0;
  // d = h 2^32 + l with a signed l: d^2 = h^2 2^64 + h l 2^33 + l^2
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int l = static_cast<int>(d[a]);
    const int h = static_cast<int>(d[a] >> 32) + static_cast<int>(static_cast<unsigned>(l) >> 31);
    H += static_cast<long long>(h) * h;
    M += static_cast<long long>(h) * l;
    lo += static_cast<unsigned>(__mulhi(l, l)) >> 2;  // three of them fit 32 bits
  }
  return (static_cast<unsigned long long>(H) << 18) + (M >> 13) + (lo >> 12);
}
// A fixed-point d2's high word (2^-24 A^2) next to that of the squared cutoff
// c2: within 6e-8 A^2, where integers and doubles differ by some 1e-14.
static __device__ __forceinline__ bool near_fix(unsigned hw, unsigned c2) { return hw - ((c2 << 24) - 1u) <= 1u; }

static __device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// Exact sum of FP64 values as a fixed-point integer with 2^-bits resolution
// (bits leaves room for the largest sum expected); values that are not finite,
// or of more than 2^(kMaxShift + 53 - bits), are kept apart in FP64.
template <int kMaxShift = 70>
struct ExactSum {
  __int128 v = 0;
  double nf = 0.0;
  __device__ __forceinline__ void add(double x, int bits) {
    const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(x));
    const int e = static_cast<int>(b >> 52) & 0x7ff;
    if (e == 0) return;  // zero (a subnormal is far below the resolution)
    const int sh = e - 1075 + bits;
    if (e == 0x7ff || sh > kMaxShift) {
      nf += x;
      return;
    }
    const unsigned long long m = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    const unsigned __int128 t = sh >= 0 ? static_cast<unsigned __int128>(m) << sh
                                        : static_cast<unsigned __int128>(m >> min(-sh, 63));
    v += static_cast<long long>(b) < 0 ? -static_cast<__int128>(t) : static_cast<__int128>(t);
  }
  // The same for the usual term, of 2^(53 - bits) to 2^(117 - bits), in some
  // two dozen instructions: the significand shifted by less than 64, two's
  // complement by the sign, one carry chain.
  __device__ __forceinline__ void add_term(double x, int bits) {
    const unsigned lo = static_cast<unsigned>(__double2loint(x)), hi = static_cast<unsigned>(__double2hiint(x));
    const int sh = static_cast<int>(hi << 1 >> 21) - 1075 + bits;
    if (static_cast<unsigned>(sh) < 64u) {
      const unsigned mh = (hi & 0xfffffu) | 0x100000u, g = static_cast<unsigned>(static_cast<int>(hi) >> 31);
      const unsigned w0 = lo << (sh & 31), w1 = __funnelshift_l(lo, mh, sh), w2 = __funnelshift_l(mh, 0u, sh);
      const bool up = (sh & 32) != 0;
      const unsigned t0 = (up ? 0u : w0) ^ g, t1 = (up ? w0 : w1) ^ g, t2 = (up ? w1 : w2) ^ g, t3 = (up ? w2 : 0u) ^ g;
      unsigned a0 = static_cast<unsigned>(v), a1 = static_cast<unsigned>(static_cast<unsigned __int128>(v) >> 32),
               a2 = static_cast<unsigned>(static_cast<unsigned __int128>(v) >> 64),
               a3 = static_cast<unsigned>(static_cast<unsigned __int128>(v) >> 96);
      asm("{\n\t.reg .u32 c;\n\tadd.cc.u32 c, %8, %8;\n\taddc.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, %5;\n\t"
          "addc.cc.u32 %2, %2, %6;\n\taddc.u32 %3, %3, %7;\n\t}"
          : "+r"(a0), "+r"(a1), "+r"(a2), "+r"(a3)
          : "r"(t0), "r"(t1), "r"(t2), "r"(t3), "r"(g));
      v = static_cast<__int128>(static_cast<unsigned __int128>(static_cast<unsigned long long>(a3) << 32 | a2) << 64 |
                                (static_cast<unsigned long long>(a1) << 32 | a0));
    } else if ((lo | hi << 1) != 0u) {
      add(x, bits);
    }
  }
  // every lane: the sum over the warp
  __device__ __forceinline__ void warp_total() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long lo = __shfl_xor_sync(kFull, static_cast<unsigned long long>(v), o);
      const long long hi = __shfl_xor_sync(kFull, static_cast<long long>(v >> 64), o);
      v += (static_cast<__int128>(hi) << 64) | lo;
    }
    if (__any_sync(kFull, __double_as_longlong(nf) != 0)) nf = warp_sum(nf);
  }
  __device__ __forceinline__ double value(int bits) const {
    const double hi = static_cast<double>(static_cast<long long>(v >> 64)),
                 lo = static_cast<double>(static_cast<unsigned long long>(v));
    const double s = ldexp(hi * 18446744073709551616.0 + lo, -bits);
    return nf != 0.0 ? nf + s : s;
  }
};

// FP32 squared distance of a receptor atom and a ligand atom (both relative to O).
static __device__ __forceinline__ float d2f(const float4 &r, float lx, float ly, float lz) {
  const float dx = __fsub_rn(r.x, lx), dy = __fsub_rn(r.y, ly), dz = __fsub_rn(r.z, lz);
  return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

// AIR energy and satisfied-restraint count (src/fitness.rs:205-267,
// src/restraints.rs:11-40) by one warp: one restraint per lane, summed in
// restraint order.
static __device__ __forceinline__ void warp_air(const ScoreParams &p, const gd_pose_frame &f, int pose, int lane,
                                                double &air, int &sat) {
  air = 0.0;
  sat = 0;
  for (int r0 = 0; r0 < p.K; r0 += 32) {
    double term = 0.0;
    int ok = 0;
    const int r = r0 + lane;
    if (r < p.K) {
      const D4 a = p.restr_rec[r];
      double X, Y, Z;
      ligand_atom(p, f, pose, p.restr_lig[r], X, Y, Z);
      const double dist = sqrt(exact_d2(a.x, a.y, a.z, X, Y, Z));
      double v = 0.0;
      if (dist < 0.0) v = __dsub_rn(0.0, dist);
      else if (dist > 7.0) v = __dsub_rn(dist, 7.0);
      term = __dmul_rn(__dmul_rn(10.0, v), v);
      ok = dist <= 7.0;
    }
    for (int k = 0; k < 32 && r0 + k < p.K; ++k) {
      air = __dadd_rn(air, __shfl_sync(kFull, term, k));
      sat += __shfl_sync(kFull, ok, k);
    }
  }
}

// Final per-pose record (src/chromosome.rs:111-127).
static __device__ __forceinline__ void write_pose(const ScoreParams &p, int pose, double vdw, double elec,
                                                  double desolv, double air, int sat) {
  const double ratio = p.K > 0 ? static_cast<double>(sat) / static_cast<double>(p.K) : 0.0;
  gd_pose_energy o;
  o.vdw = vdw;
  o.elec = elec;
  o.desolv = desolv;
  o.air = air;
  o.restraint_penalty = __dmul_rn(__dsub_rn(1.0, ratio), static_cast<double>(p.K));
  o.fitness = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(p.wv, vdw), __dmul_rn(p.we, elec)), __dmul_rn(p.wd, desolv)),
                        __dmul_rn(p.wa, air));
  p.out[pose] = o;
}

}  // namespace gd
