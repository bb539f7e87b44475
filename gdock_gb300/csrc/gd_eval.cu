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
// pose's ligand atoms; per atom the difference from its partner is one chain
// of fused multiply-adds, the distance its square root, the sums exact integer
// ones; contacts are decided in FP32 outside a guard band and exactly (the
// reference's transform and threshold) inside it, and distances that
// cancellation would spoil (below 1/4 A) are redone in the reference's order.
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

struct gd_evaluator {
  gd_complex *cx = nullptr;
  gd_context *ctx = nullptr;
  int n_u = 0;                            // ligand atoms the metrics read
  int n_ref = 0, n_iref = 0, n_native = 0;  // divisors: |reference|, |reference interface|, |native contacts|
  int n_p = 0;                            // native-identity (receptor atom, ligand atom) pairs
  int64_t counts[GD_EVAL_COUNTS] = {};    // as gd_evaluator_counts reports them
  const int *u_slot = nullptr;            // [n_u] device slot of each such ligand atom (interface atoms first)
  int n_if = 0;                           // the first n_if of them have an i-RMSD partner or native contacts
  const D4 *u_x0 = nullptr;               // [n_u] ligand atom relative to the rotation centre
  const D4 *u_ref = nullptr;              // [n_u] paired reference atom (w = 1) or none (w = 0)
  const D4 *u_iref = nullptr;             // [n_if] likewise; w = 2: the same atom as u_ref
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
  const D4 *u_x0, *u_ref, *u_iref, *p_rec;
  const float4 *p_rec32;
  int n_u, n_if, n_ref, n_iref, n_native;
  double thr5;
  float extent;     // bounds |coordinate - O| of receptor and ligand atoms before the displacement
  const int *skip;  // nonzero: no work (a finished GA job); may be null
  gd_dock_metrics *out;
};

constexpr int kEvalWarps = 8;
constexpr int kEvalCtas = 2;    // resident per SM (registers)
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

// sqrt(d2) for d2 in [1/16, 2^900): s (1 - e)^(-1/2) by its Taylor series to
// the second order on the hardware's approximation y of d2^(-1/2), with
// s = d2 y and e = 1 - s y (about 2^-20, so that the next term lies below the
// FP64 rounding): five FP64 operations.
__device__ __forceinline__ double sqrt64(double d2) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d2));
  const double s = d2 * y, e = __fma_rn(-s, y, 1.0);
  return __fma_rn(s, e * __fma_rn(e, 0.375, 0.5), s);
}

// What bounds it: the FP64 pipe.  The reference's transform, difference,
// square and correctly rounded root cost about 60 FP64 operations per atom;
// this form takes 12 for the difference, 3 and 5 for square and root and adds
// in integers.  WPP warps per pose: one where the poses fill the GPU, else the
// whole CTA (150 poses of one warp each kept 38 of the 152 SMs waiting on
// FP64 latency).
// 65,536 poses of 2,538 x 1,280 atoms (the whole call, host frames and copies
// included) 10.8 -> 4.32 ms; the kernel on 150 poses of 1,074 x 741 atoms 99 ->
// 18 us.
template <int WPP>
__global__ void __launch_bounds__(kEvalWarps * 32, kEvalCtas) k_dockq(const EvalParams e) {
  if (e.skip && *e.skip) return;
  __shared__ gd_pose_frame s_f[kEvalWarps / WPP];
  __shared__ __int128 s_sum[kEvalWarps][2];
  __shared__ double s_nf[kEvalWarps][2];
  __shared__ int s_common[kEvalWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int step = gridDim.x * (kEvalWarps / WPP);
  const int t0 = WPP == 1 ? lane : static_cast<int>(threadIdx.x);
  gd_pose_frame &f = s_f[WPP == 1 ? warp : 0];
  // lane k keeps the k-th pose's sums until the warp has 32 of them: the
  // divisions and roots of the metrics then run on all lanes
  DistSum my_l, my_i;
  int my_common = 0, my_pose = -1, held = 0;
  auto finish = [&]() {
    if (my_pose >= 0) {
      // src/evaluator.rs:68-84, without contraction into fused multiply-adds
      const double sl = my_l.value(kDistBits), si = my_i.value(kDistBits);
      const double rmsd = e.n_ref ? __dsqrt_rn(__ddiv_rn(sl, static_cast<double>(e.n_ref))) : 0.0;
      const double irmsd = e.n_iref ? __dsqrt_rn(__ddiv_rn(si, static_cast<double>(e.n_iref))) : 0.0;
      const double fnat = e.n_native ? __ddiv_rn(static_cast<double>(my_common), static_cast<double>(e.n_native)) : 0.0;
      const double a = __ddiv_rn(irmsd, 1.5), b = __ddiv_rn(rmsd, 8.5);
      const double is = __ddiv_rn(1.0, __dadd_rn(1.0, __dmul_rn(a, a)));
      const double ls = __ddiv_rn(1.0, __dadd_rn(1.0, __dmul_rn(b, b)));
      const double dockq = __ddiv_rn(__dadd_rn(__dadd_rn(fnat, is), ls), 3.0);
      e.out[my_pose] = gd_dock_metrics{rmsd, irmsd, fnat, dockq};
    }
    my_pose = -1;
    held = 0;
  };
  for (int pose = blockIdx.x * (kEvalWarps / WPP) + (WPP == 1 ? warp : 0); pose < e.p.n_poses; pose += step) {
    if (WPP == 1) __syncwarp();
    else __syncthreads();
    if (t0 < 16) reinterpret_cast<double *>(&f)[t0] = reinterpret_cast<const double *>(e.p.frames + pose)[t0];
    if (WPP == 1) __syncwarp();
    else __syncthreads();
    // moved atom = R x0 + (centre + displacement)
    const double m00 = f.ca * f.cb, m01 = f.m01, m02 = f.m02, m10 = f.sa * f.cb, m11 = f.m11, m12 = f.m12;
    const double m20 = -f.sb, m21 = f.cb * f.sg, m22 = f.cb * f.cg;
    const double tx = e.p.cx + f.dx, ty = e.p.cy + f.dy, tz = e.p.cz + f.dz;
    // the FP32 guard band of the contact test, as for the contact bitmaps
    // (M bounds the coordinates; twice it covers the sum that forms them)
    const float M = 2.0f * (e.extent + fmaxf(fabsf(static_cast<float>(f.dx)),
                                             fmaxf(fabsf(static_cast<float>(f.dy)), fabsf(static_cast<float>(f.dz)))));
    const float guard = 4.0f * (17.33f * (2.0f * M + 5.0f) + 100.0f) * 0x1p-24f + 1e-6f;
    const bool band_ok = guard < 1.0f;
    DistSum sl, si;
    int common = 0;
#pragma unroll 1
    for (int u = t0; u < e.n_u; u += 32 * WPP) {
      const D4 a = e.u_x0[u], r = e.u_ref[u];
      auto from = [&](const D4 &q, double &dx, double &dy, double &dz) {
        dx = __fma_rn(m00, a.x, __fma_rn(m01, a.y, __fma_rn(m02, a.z, tx - q.x)));
        dy = __fma_rn(m10, a.x, __fma_rn(m11, a.y, __fma_rn(m12, a.z, ty - q.y)));
        dz = __fma_rn(m20, a.x, __fma_rn(m21, a.y, __fma_rn(m22, a.z, tz - q.z)));
      };
      auto distance = [&](const D4 &q, double dx, double dy, double dz) {
        const double d2 = __fma_rn(dz, dz, __fma_rn(dy, dy, dx * dx));
        const int hi = __double2hiint(d2);
        if (hi < 0x3fb00000 || hi >= 0x78300000) {  // below 1/16, or from 2^900 (and NaN) on
          int slot = e.u_slot[u];
          if (!GD_DCHECK(e.p.err, slot >= 0 && slot < e.p.nl, 40)) slot = 0;
          return exact_distance(e.p, f, pose, slot, q.x, q.y, q.z);
        }
        return sqrt64(d2);
      };
      double dx, dy, dz;
      from(r, dx, dy, dz);
      double d = 0.0;
      if (r.w != 0.0) {
        d = distance(r, dx, dy, dz);
        sl.add(d, kDistBits);
      }
      if (u < e.n_if) {
        const D4 q = e.u_iref[u];
        if (q.w == 2.0) {
          si.add(d, kDistBits);
        } else if (q.w != 0.0) {
          double ex, ey, ez;
          from(q, ex, ey, ez);
          si.add(distance(q, ex, ey, ez), kDistBits);
        }
        int k = e.u_pbeg[u];
        const int k1 = e.u_pbeg[u + 1];
        if (k < k1) {
          const float lx = static_cast<float>(dx) + static_cast<float>(r.x - e.p.ox),
                      ly = static_cast<float>(dy) + static_cast<float>(r.y - e.p.oy),
                      lz = static_cast<float>(dz) + static_cast<float>(r.z - e.p.oz);
          for (; k < k1; ++k) {
            const float t = d2f(__ldg(&e.p_rec32[k]), lx, ly, lz) - 25.0f;
            bool hit = t < 0.0f;
            if (!(band_ok && fabsf(t) > guard)) {
              int slot = e.u_slot[u];
              if (!GD_DCHECK(e.p.err, slot >= 0 && slot < e.p.nl, 40)) slot = 0;
              hit = exact_contact(e.p, f, pose, slot, e.p_rec[k], e.thr5);
            }
            common += hit;
          }
        }
      }
    }
    sl.warp_total();
    si.warp_total();
    common = __reduce_add_sync(kFull, common);
    if (WPP > 1) {
      if (lane == 0) {
        s_sum[warp][0] = sl.v;
        s_sum[warp][1] = si.v;
        s_nf[warp][0] = sl.nf;
        s_nf[warp][1] = si.nf;
        s_common[warp] = common;
      }
      __syncthreads();
      if (warp == 0) {
        for (int w = 1; w < WPP; ++w) {
          sl.v += s_sum[w][0];
          si.v += s_sum[w][1];
          sl.nf += s_nf[w][0];
          si.nf += s_nf[w][1];
          common += s_common[w];
        }
      }
    }
    if (WPP == 1 || warp == 0) {
      if (lane == held) {
        my_l = sl;
        my_i = si;
        my_common = common;
        my_pose = pose;
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
  ep.u_x0 = ev->u_x0;
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
  // one warp per pose when the poses give every resident warp one, else a CTA
  // per pose
  const int warps = kEvalCtas * kEvalWarps * ev->ctx->sm_count;
  if (n >= warps)
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
  std::vector<D4> u_x0(nu), u_ref(nu), u_iref(n_if), p_rec;
  std::vector<float4> p_rec32;
  p_rec.reserve(n_p);
  p_rec32.reserve(n_p);
  for (int u = 0; u < nu; ++u) {
    const int j = order[u];
    u_slot[u] = cx->h_lig_slot[j];
    u_x0[u] = D4{cx->h_lx[j] - cx->cx, cx->h_ly[j] - cx->cy, cx->h_lz[j] - cx->cz, 0.0};
    u_ref[u] = l_ref[j];
    if (u >= n_if) continue;
    u_iref[u] = l_iref[j];
    if (l_ref[j].w != 0.0 && l_iref[j].w != 0.0 && l_ref[j].x == l_iref[j].x && l_ref[j].y == l_iref[j].y &&
        l_ref[j].z == l_iref[j].z)
      u_iref[u].w = 2.0;
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
  ev->thr5 = make_thresholds(5.0).contact_le;
  const int64_t cnt[GD_EVAL_COUNTS] = {static_cast<int64_t>(rec_if.size()), static_cast<int64_t>(ref_if.size()),
                                       n_native, nu, std::min(nl, nf),
                                       static_cast<int64_t>(std::min(lig_i.size(), ref_i.size())), n_p};
  std::copy(cnt, cnt + GD_EVAL_COUNTS, ev->counts);
  auto al = [](size_t b) { return (std::max<size_t>(b, 1) + 255) / 256 * 256; };
  const size_t b_slot = al(sizeof(int) * nu), b_beg = al(sizeof(int) * (n_if + 1)), b_ref = al(sizeof(D4) * nu),
               b_iref = al(sizeof(D4) * n_if), b_prec = al(sizeof(D4) * p_rec.size()),
               b_prec32 = al(sizeof(float4) * p_rec32.size());
  ev->bytes = b_slot + b_beg + 2 * b_ref + b_iref + b_prec + b_prec32;
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
  ev->u_x0 = reinterpret_cast<const D4 *>(put(u_x0.data(), sizeof(D4) * nu, b_ref));
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
  gd_status s = ensure_scratch(ctx, fb_al + ob, staged ? fb_al + ob : 0);
  if (s != GD_OK) return s;
  gd_pose_frame *d_frames = static_cast<gd_pose_frame *>(ctx->d_scratch);
  gd_dock_metrics *d_out = reinterpret_cast<gd_dock_metrics *>(static_cast<char *>(ctx->d_scratch) + fb_al);
  std::vector<gd_pose_frame> pageable(staged ? 0 : n);
  gd_pose_frame *frames = staged ? static_cast<gd_pose_frame *>(ctx->h_pinned) : pageable.data();
  void *res = staged ? static_cast<char *>(ctx->h_pinned) + fb_al : static_cast<void *>(out);
  gd_make_frames(genes, n, frames);
  cudaStream_t st = ctx->stream;
  cudaError_t e = cudaMemcpyAsync(d_frames, frames, fb, cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "evaluator frames upload");
  s = gd_evaluate_frames_device(ev, d_frames, n, d_out, st);
  if (s == GD_OK) {
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
