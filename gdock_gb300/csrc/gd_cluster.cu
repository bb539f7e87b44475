// FCC clustering: residue contacts per pose, all-pairs fraction of common
// contacts by popcount, neighbour graph, greedy clustering.
//
// Reference: src/clustering.rs:62-293.  Residues are keyed by (chain,
// resseq) over non-hydrogen atoms of the receptor+ligand complex; a contact
// is a pair of residues on different chains with an atom pair at distance
// <= cutoff; FCC(i,j) = |Xi & Xj| / |Xi| (and / |Xj|), an edge i->j when
// FCC >= c and FCC_v >= c * strictness; greedy clustering picks the element
// with most unused neighbours (ties: lower index).
//
// GPU pieces:
//   k_contacts     a CTA per (pose, part): warps take blocks of ligand residues,
//                  cull receptor residues by bounding spheres, test the near
//                  residue pairs' atoms in FP32 (FP64 next to the cutoff) and
//                  append the contacts to the pose's list and to the union.
//   k_contacts_rl  the same lists with every atom pair decided in FP64, for
//                  topologies k_contacts does not take.
//   k_rows, k_fcc  the lists as bitsets over the compacted union; tiles of pose
//                  pairs, AND + popcount; the reference's FP64 ratio tests.
//   k_post_*       the pair counts from per-contact pose lists instead, for
//                  contacts spread thin.
//   k_greedy       the greedy clustering over the adjacency bit matrix.
// Host pieces: key canonicalisation (smaller chain first), receptor-only and
// ligand-only inter-chain contacts of multi-chain molecules, the universe of
// caller-supplied sets, and the output order.
#include <cooperative_groups.h>

#include <algorithm>
#include <chrono>
#include <iterator>
#include <cmath>
#include <cstring>
#include <map>
#include <functional>
#include <numeric>
#include <thread>
#include <vector>

#include "gd_device.cuh"

namespace gd {

namespace cg = cooperative_groups;

struct ClusterTopo {
  // receptor heavy atoms grouped by residue (canonical ids), ligand likewise
  int GR = 0, GL = 0;
  std::vector<int64_t> rg_key, lg_key;  // (chain << 16) | uint16(resseq)
  std::vector<int> rg_rank, lg_rank;    // the keys' ranks among their molecule's
  std::vector<int> rg_off, lg_off;      // atom ranges
  std::vector<int> r_atoms, l_atoms;    // original atom indices, grouped
  // the residues of a molecule of several chains in the order of their keys, for
  // the contacts within it
  struct Groups {
    std::vector<int64_t> key;
    std::vector<int> off, atoms;
  } r_by_key, l_by_key;
  bool multi_chain_rec = false, multi_chain_lig = false;
  bool mixed = false;  // a (chain, resseq) residue with atoms in both molecules
  float4 *d_r32 = nullptr;  // receptor heavy atoms (x-O, y-O, z-O, 0) FP32, grouped
  std::vector<int64_t> rr_keys;         // receptor-only inter-chain contacts (pose independent)
  double rr_cutoff = -1.0;
  // ligand-only inter-chain contacts in the positioned frame: their count,
  // and whether some residue pair's closest atom pair lies so near the cutoff
  // that FP64 rounding of a pose's transform could flip it (then the count is
  // not pose independent and the per-pose host path decides)
  long long ll_count = 0;
  bool ll_unstable = false;
  double ll_cutoff = -1.0;
  // device
  double *d_rx = nullptr, *d_ry = nullptr, *d_rz = nullptr;
  double *d_lx = nullptr, *d_ly = nullptr, *d_lz = nullptr;
  int *d_rg_off = nullptr, *d_lg_off = nullptr;
  float4 *d_rg_sph = nullptr;   // (centre - O, radius) FP32
  float4 *d_rb_sph = nullptr;   // per 32 consecutive receptor residues: sphere enclosing theirs
  D4 *d_lg_sph = nullptr;  // (centre in the positioned frame, radius)
  float4 *d_lg_rel = nullptr, *d_lb_rel = nullptr;  // spheres relative to the rotation centre: per ligand residue, per
                                                    // block of kLigBlock of them
  D4 *d_l_rel = nullptr;   // ligand heavy atoms relative to the rotation centre, grouped
  uint8_t *d_rg_chain = nullptr, *d_lg_chain = nullptr;
  std::vector<void *> allocs;
  uint64_t bytes = 0;
};

namespace {

constexpr int kMaxGroupAtoms = 64;

// Under GD_TRACE: wait for the stream and print the time since `t` (then
// reset it), so that device phases can be told apart.  No-op otherwise.
void trace_step(const char *name, cudaStream_t st, std::chrono::steady_clock::time_point &t) {
  if (!trace_on()) return;
  cudaStreamSynchronize(st);
  const auto now = std::chrono::steady_clock::now();
  trace(name, std::chrono::duration<double>(now - t).count());
  t = now;
}

struct PhaseTimer {
  const char *name;
  std::chrono::steady_clock::time_point t0 = std::chrono::steady_clock::now();
  explicit PhaseTimer(const char *n) : name(n) {}
  ~PhaseTimer() { trace(name, std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count()); }
};

struct ContactParams {
  const double *rx, *ry, *rz;
  const int *rg_off;
  const float4 *rg_sph;
  const uint8_t *rg_chain;
  const double *lx, *ly, *lz;
  const int *lg_off;
  const D4 *lg_sph;
  const uint8_t *lg_chain;
  int GR, GL;
  double cx, cy, cz, ox, oy, oz;
  const gd_pose_frame *frames;
  int n;
  double t_le;     // contact decision: d2 <= t_le
  float reach;     // cutoff + culling margin
  int *counts;     // [n]
  uint32_t *lists; // [n * cap]
  int cap;
};

constexpr int kContactWarps = 4;
constexpr int kLigBlock = 8;    // ligand residues of a block (one enclosing sphere)
constexpr int kCandMax = 1024;  // receptor residue candidates kept per unit
constexpr int kUnitAtoms = 128;   // ligand atoms of a unit moved in one pass (else residue by residue)
constexpr int kNearMax = 128;   // near residue pairs listed before they are tested
constexpr int kOutMax = 64;     // contacts a warp holds before it appends them

__global__ void __launch_bounds__(kContactWarps * 32) k_contacts_rl(const ContactParams p) {
  __shared__ double s_xyz[kContactWarps][3][kMaxGroupAtoms];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const long long items = static_cast<long long>(p.n) * p.GL;
  for (long long it = static_cast<long long>(blockIdx.x) * kContactWarps + wib; it < items;
       it += static_cast<long long>(gridDim.x) * kContactWarps) {
    const int pose = static_cast<int>(it / p.GL), lg = static_cast<int>(it % p.GL);
    const gd_pose_frame f = p.frames[pose];
    const int a0 = p.lg_off[lg], na = p.lg_off[lg + 1] - a0;
    const bool staged = na <= kMaxGroupAtoms;
    if (staged) {
      for (int a = lane; a < na; a += 32) {
        double X, Y, Z;
        transform_atom(f, p.cx, p.cy, p.cz, p.lx[a0 + a], p.ly[a0 + a], p.lz[a0 + a], X, Y, Z);
        s_xyz[wib][0][a] = X;
        s_xyz[wib][1][a] = Y;
        s_xyz[wib][2][a] = Z;
      }
    }
    __syncwarp();
    // culling sphere of the ligand residue after the transform
    const D4 ls = p.lg_sph[lg];
    double CX, CY, CZ;
    transform_atom(f, p.cx, p.cy, p.cz, ls.x, ls.y, ls.z, CX, CY, CZ);
    const float lcx = static_cast<float>(CX - p.ox), lcy = static_cast<float>(CY - p.oy),
                lcz = static_cast<float>(CZ - p.oz);
    const float lrad = static_cast<float>(ls.w);
    const uint8_t lchain = p.lg_chain[lg];
    for (int rg = lane; rg < p.GR; rg += 32) {
      if (p.rg_chain[rg] == lchain) continue;
      const float4 rs = p.rg_sph[rg];
      const float dx = rs.x - lcx, dy = rs.y - lcy, dz = rs.z - lcz;
      const float lim = rs.w + lrad + p.reach;
      if (dx * dx + dy * dy + dz * dz > lim * lim) continue;
      bool found = false;
      for (int b = p.rg_off[rg]; b < p.rg_off[rg + 1] && !found; ++b) {
        const double bx = p.rx[b], by = p.ry[b], bz = p.rz[b];
        for (int a = 0; a < na; ++a) {
          double X, Y, Z;
          if (staged) {
            X = s_xyz[wib][0][a];
            Y = s_xyz[wib][1][a];
            Z = s_xyz[wib][2][a];
          } else {
            transform_atom(f, p.cx, p.cy, p.cz, p.lx[a0 + a], p.ly[a0 + a], p.lz[a0 + a], X, Y, Z);
          }
          if (exact_d2(bx, by, bz, X, Y, Z) <= p.t_le) {
            found = true;
            break;
          }
        }
      }
      if (found) {
        const int slot = atomicAdd(&p.counts[pose], 1);
        if (slot < p.cap) p.lists[static_cast<size_t>(pose) * p.cap + slot] = static_cast<uint32_t>(rg) * p.GL + lg;
      }
    }
    __syncwarp();
  }
}

// ---- FCC pair decisions ----

// The ratio tests of calculate_fcc (src/clustering.rs:122-132) and
// create_elements (src/clustering.rs:171) for one pose pair: bit 0 edge
// i -> j, bit 1 edge j -> i (the same ratios, roles swapped).  Out of line:
// only pairs next to a threshold come here.
__device__ __noinline__ int fcc_edges_exact(int common, int si, int sj, double c, double cs) {
  const double m = static_cast<double>(common);
  const double fcc = m / static_cast<double>(si), fcc_v = m / static_cast<double>(sj);
  return (fcc >= c && fcc_v >= cs) | (fcc_v >= c && fcc >= cs) << 1;
}

// The same from FP32 ratios where all four comparisons are clear of their
// threshold by 1e-5 (1 + |threshold|), far above FP32 rounding.  In FP64 alone
// the divisions of every pair kept the FP64 pipe 72 % busy (0.90 ms of 4,096
// poses' pair counts).
__device__ __forceinline__ int fcc_edges(int common, int si, int sj, double c, double cs, float c32, float cs32) {
  if (si <= 0 || sj <= 0) return 0;
  const float m = static_cast<float>(common);
  const float a = m * rcp_approx(static_cast<float>(si)), b = m * rcp_approx(static_cast<float>(sj));
  const float mc = 1e-5f * (1.0f + fabsf(c32)), ms = 1e-5f * (1.0f + fabsf(cs32));
  const bool clear = fabsf(a - c32) > mc && fabsf(b - c32) > mc && fabsf(a - cs32) > ms && fabsf(b - cs32) > ms;
  if (!clear) return fcc_edges_exact(common, si, sj, c, cs);
  return (a > c32 && b > cs32) | (b > c32 && a > cs32) << 1;
}

// pose bitsets over the compacted contact universe: rows of 64-bit words
struct FccParams {
  const unsigned long long *bits;
  const int *sizes;
  const int *info;  // info[0]: contacts of the universe
  int n, stride;    // poses; words a row has room for
  double c, cs;     // fcc_cutoff and fcc_cutoff * strictness
  uint32_t *adj;    // n rows of ceil(n/32) words; bit j of row i: edge i -> j
  int adj_words;
  int c0;           // contacts every pose has (inter-chain ones within one molecule), not in the bitsets
};

constexpr int kFW = 18;   // words per staged chunk (groups of 3; row stride 19 words: no bank conflicts)

// T x T pose pairs per CTA, T/16 x T/16 per thread.  The common count of a
// pose pair is symmetric: only tiles on or above the diagonal run, and an
// off-diagonal tile decides both directions of each pair.  The edge bits of a
// tile are collected in shared memory and stored as whole (half) words.
template <int T>
__global__ void __launch_bounds__(256) k_fcc(const FccParams p) {
  if (blockIdx.y > blockIdx.x) return;
  constexpr int Q = T / 16;
  __shared__ unsigned long long sa[T][kFW + 1];
  __shared__ unsigned long long sb[T][kFW + 1];
  __shared__ uint32_t s_edge[2][T][2];  // forward rows i, backward rows j
  const int i0 = blockIdx.y * T, j0 = blockIdx.x * T;
  const bool diag = blockIdx.y == blockIdx.x;
  const int W = (p.info[0] + 63) / 64;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;  // 16 x 16 threads, Q x Q pairs each
  for (int e = threadIdx.x; e < 4 * T; e += 256) (&s_edge[0][0][0])[e] = 0;
  int cnt[Q][Q];
#pragma unroll
  for (int a = 0; a < Q; ++a)
#pragma unroll
    for (int b = 0; b < Q; ++b) cnt[a][b] = 0;
  for (int w0 = 0; w0 < W; w0 += kFW) {
    for (int e = threadIdx.x; e < T * kFW; e += 256) {
      const int r = e / kFW, w = e % kFW;
      const int gi = i0 + r, gj = j0 + r, gw = w0 + w;
      sa[r][w] = (gi < p.n && gw < W) ? p.bits[static_cast<size_t>(gi) * p.stride + gw] : 0ull;
      sb[r][w] = (gj < p.n && gw < W) ? p.bits[static_cast<size_t>(gj) * p.stride + gw] : 0ull;
    }
    __syncthreads();
    // three words at a time through a carry-save step: with l = x0^x1^x2 and
    // h = majority(x0, x1, x2), popc(x0) + popc(x1) + popc(x2) =
    // 2 popc(h) + popc(l): two popcounts (the XU pipe) instead of three
    // (seven words through full adders took 0.85 ms instead of 0.77 on 4,096
    // poses: the logic pipe binds)
#pragma unroll 1
    for (int w = 0; w < kFW; w += 3) {
      unsigned long long av[Q][3], bv[Q][3];
#pragma unroll
      for (int a = 0; a < Q; ++a)
#pragma unroll
        for (int i = 0; i < 3; ++i) av[a][i] = sa[ty + 16 * a][w + i];
#pragma unroll
      for (int b = 0; b < Q; ++b)
#pragma unroll
        for (int i = 0; i < 3; ++i) bv[b][i] = sb[tx + 16 * b][w + i];
#pragma unroll
      for (int a = 0; a < Q; ++a)
#pragma unroll
        for (int b = 0; b < Q; ++b) {
          const unsigned long long x0 = av[a][0] & bv[b][0], x1 = av[a][1] & bv[b][1], x2 = av[a][2] & bv[b][2];
          const unsigned long long l = x0 ^ x1 ^ x2, h = (x0 & x1) | (x2 & (x0 ^ x1));
          cnt[a][b] += 2 * __popcll(h) + __popcll(l);
        }
    }
    __syncthreads();
  }
  if (W == 0) __syncthreads();  // s_edge is cleared
  const float c32 = static_cast<float>(p.c), cs32 = static_cast<float>(p.cs);
#pragma unroll
  for (int a = 0; a < Q; ++a) {
    const int r = ty + 16 * a, i = i0 + r;
    const int si = i < p.n ? p.sizes[i] + p.c0 : 0;
#pragma unroll
    for (int b = 0; b < Q; ++b) {
      const int c = tx + 16 * b, j = j0 + c;
      const int sj = j < p.n ? p.sizes[j] + p.c0 : 0;
      const int e = fcc_edges(cnt[a][b] + p.c0, si, sj, p.c, p.cs, c32, cs32);
      if (e & 1) atomicOr(&s_edge[0][r][c >> 5], 1u << (c & 31));
      if (e & 2) atomicOr(&s_edge[1][c][r >> 5], 1u << (r & 31));
    }
  }
  __syncthreads();
  // rows [i0, i0 + T) x columns [j0, j0 + T), then the mirrored tile
  for (int e = threadIdx.x; e < 2 * T; e += 256) {
    const int side = e / T, r = e % T;
    if (side && diag) break;
    const int row = (side ? j0 : i0) + r, col = side ? i0 : j0;
    if (row >= p.n) continue;
    uint32_t *out = p.adj + static_cast<size_t>(row) * p.adj_words + (col >> 5);
    if (T == 16) {
      reinterpret_cast<uint16_t *>(out)[(col >> 4) & 1] = static_cast<uint16_t>(s_edge[side][r][0]);
    } else {
#pragma unroll
      for (int w = 0; w < T / 32; ++w)
        if ((col >> 5) + w < p.adj_words) out[w] = s_edge[side][r][w];
    }
  }
}

cudaError_t launch_fcc(const FccParams &p, cudaStream_t st) {
  // small launches in small tiles, to fill the SMs (whole calls on 1,074 x 741
  // atoms, tiles of 16 / 64: 183 poses 138 / 150 us, 1,024 poses 337 / 349,
  // 2,048 poses 560 / 552; the kernel on 183 poses 68 -> 7 us)
  // Every word of the matrix is stored by some tile (tiles of 16 go on to a
  // whole word), so it is not cleared first.
  const int T = p.n <= 1024 ? 16 : 64, tiles = T == 16 ? 2 * p.adj_words : (p.n + T - 1) / T;
  const dim3 grid(tiles, tiles);
  if (T == 16) k_fcc<16><<<grid, 256, 0, st>>>(p);
  else k_fcc<64><<<grid, 256, 0, st>>>(p);
  return cudaGetLastError();
}

__global__ void k_compact_lists(const uint32_t *lists, const int *counts, const long long *offs, int n, int cap,
                                uint32_t *out) {
  for (long long pose = blockIdx.x; pose < n; pose += gridDim.x) {
    const int c = min(counts[pose], cap);
    for (int k = threadIdx.x; k < c; k += blockDim.x) out[offs[pose] + k] = lists[pose * cap + k];
  }
}

// ---- contact lists on the device ----

struct ContactListParams {
  const float4 *r32;
  const double *rx, *ry, *rz;
  const int *rg_off;
  const float4 *rg_sph, *rb_sph;
  const uint8_t *rg_chain;
  const double *lx, *ly, *lz;
  const int *lg_off;
  const D4 *l_rel;
  const float4 *lg_rel, *lb_rel;
  const uint8_t *lg_chain;
  int GR, GL;
  double cx, cy, cz, ox, oy, oz;
  const gd_pose_frame *frames;
  int parts, unit;   // CTAs per pose; ligand residues per unit (divides kLigBlock)
  double t_le;       // exact decision d2 <= t_le
  float t32, guard;  // FP32 decision d2 <= t32 outside |d2 - t32| < guard
  float reach;
  int *counts;       // [n] contacts found (beyond cap too)
  uint32_t *lists;   // [n][cap], entries rg * GL + lg in any order
  int cap;
  uint32_t *ubits;   // union of all poses' contacts, bit rg * GL + lg; may be null
  uint32_t *rows;    // [n][row_words] each pose's contacts, the same bits; may be null
  long long row_words;
  int *err;          // the context's error word (index checks of the debug library)
};

// Exact re-decision of a pair in the guard band: the ligand atom moved in the
// reference's order, its distance order.  Out of line: rare.
__device__ __noinline__ bool exact_contact(const ContactListParams &p, int pose, int b, int a) {
  double X, Y, Z;
  transform_atom(p.frames[pose], p.cx, p.cy, p.cz, p.lx[a], p.ly[a], p.lz[a], X, Y, Z);
  return exact_d2(p.rx[b], p.ry[b], p.rz[b], X, Y, Z) <= p.t_le;
}

// Warps take units of `unit` consecutive ligand residues.  Per unit: the
// residues' and the block's spheres moved; receptor residues within reach of
// the block (groups of 32 first) listed as candidates; each ligand residue's
// near ones listed as residue pairs; the pairs tested two at a time, one per
// half warp: the receptor atoms that reach the ligand residue's sphere against
// its atoms, one per lane, until the first contact.  The unit's atoms are moved
// once it has a near pair.
// What bounds it: instruction issue.  The former kernel (whole warps per
// residue pair, every block's atoms moved in the reference's 34 FP64
// operations) kept the FP64 pipe 77 % busy and wrote bitmaps over all residue
// pairs, whose clearing, union and compaction moved 2 GB for 4,096 poses of
// 2,000 x 500 residues: contacts and union 3.0 -> 0.81 ms.
__global__ void __launch_bounds__(kContactWarps * 32) k_contacts(const ContactListParams p) {
  __shared__ double s_m[12];  // rotation by rows, then centre + displacement - O
  __shared__ float s_m32[12];
  __shared__ int s_next;
  __shared__ float4 s_f[kContactWarps][kUnitAtoms];       // the unit's moved atoms (FP32, relative to O)
  __shared__ float4 s_ls[kContactWarps][kLigBlock + 1];   // its residues' spheres, then the block's
  __shared__ uint16_t s_cand[kContactWarps][kCandMax];
  __shared__ uint32_t s_near[kContactWarps][kNearMax + 32];  // receptor residue | unit residue << 16
  __shared__ uint32_t s_out[kContactWarps][kOutMax];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, half = lane >> 4, l16 = lane & 15;
  const unsigned lt_mask = (1u << lane) - 1u;
  const int pose = static_cast<int>(blockIdx.x) / p.parts, part = static_cast<int>(blockIdx.x) % p.parts;
  if (threadIdx.x < 12) {
    const gd_pose_frame &f = p.frames[pose];
    const int k = threadIdx.x;
    const double a[] = {f.ca, f.m01, f.m02, f.sa, f.m11, f.m12, -f.sb, f.cb, f.cb, p.cx, p.cy, p.cz};
    const double b[] = {f.cb, 1.0, 1.0, f.cb, 1.0, 1.0, 1.0, f.sg, f.cg, f.dx, f.dy, f.dz};
    const double o[] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, p.ox, p.oy, p.oz};
    const double v = k < 9 ? a[k] * b[k] : (a[k] + b[k]) - o[k];
    s_m[k] = v;
    s_m32[k] = static_cast<float>(v);
  }
  if (threadIdx.x == 0) s_next = 0;
  __syncthreads();
  // atoms in FP64, rounded; spheres in FP32 (the reach has room for it)
  auto move = [&](const D4 &v) {
    return make_float4(
        static_cast<float>(__fma_rn(s_m[0], v.x, __fma_rn(s_m[1], v.y, __fma_rn(s_m[2], v.z, s_m[9])))),
        static_cast<float>(__fma_rn(s_m[3], v.x, __fma_rn(s_m[4], v.y, __fma_rn(s_m[5], v.z, s_m[10])))),
        static_cast<float>(__fma_rn(s_m[6], v.x, __fma_rn(s_m[7], v.y, __fma_rn(s_m[8], v.z, s_m[11])))), 0.0f);
  };
  auto move32 = [&](const float4 &v) {
    return make_float4(s_m32[0] * v.x + s_m32[1] * v.y + s_m32[2] * v.z + s_m32[9],
                       s_m32[3] * v.x + s_m32[4] * v.y + s_m32[5] * v.z + s_m32[10],
                       s_m32[6] * v.x + s_m32[7] * v.y + s_m32[8] * v.z + s_m32[11], v.w);
  };
  auto within = [&](const float4 &a, const float4 &b) {
    const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z, lim = a.w + b.w + p.reach;
    return dx * dx + dy * dy + dz * dz <= lim * lim;
  };
  int nout = 0;
  auto flush = [&]() {
    __syncwarp();
    int at = 0;
    if (lane == 0) at = atomicAdd(&p.counts[pose], nout);
    at = __shfl_sync(kFull, at, 0);
    for (int k = lane; k < nout; k += 32) {
      const uint32_t v = s_out[wib][k];
      if (at + k < p.cap) p.lists[static_cast<size_t>(pose) * p.cap + at + k] = v;
      if (p.ubits) atomicOr(&p.ubits[v >> 5], 1u << (v & 31));
      if (p.rows) atomicOr(&p.rows[pose * p.row_words + (v >> 5)], 1u << (v & 31));
    }
    __syncwarp();
    nout = 0;
  };
  const int nunit = (p.GL + p.unit - 1) / p.unit, nrb = (p.GR + 31) / 32;
  for (;;) {
    int u = 0;
    if (lane == 0) u = atomicAdd(&s_next, 1);
    u = __shfl_sync(kFull, u, 0) * p.parts + part;
    if (u >= nunit) break;
    const int lg0 = u * p.unit, lg1 = min(p.GL, lg0 + p.unit);
    if (lane < lg1 - lg0) s_ls[wib][lane] = move32(p.lg_rel[lg0 + lane]);
    else if (lane == kLigBlock) s_ls[wib][kLigBlock] = move32(p.lb_rel[lg0 / kLigBlock]);
    __syncwarp();
    int ncand = 0;
    {
      const float4 bs = s_ls[wib][kLigBlock];
      for (int g0 = 0; g0 < nrb; g0 += 32) {
        unsigned groups = __ballot_sync(kFull, g0 + lane < nrb && within(p.rb_sph[min(g0 + lane, nrb - 1)], bs));
        while (groups) {
          const int rg = (g0 + __ffs(groups) - 1) * 32 + lane;
          groups &= groups - 1;
          const bool near = rg < p.GR && within(p.rg_sph[min(rg, p.GR - 1)], bs);
          const unsigned m = __ballot_sync(kFull, near);
          const int pos = ncand + __popc(m & lt_mask);
          if (near && pos < kCandMax) s_cand[wib][pos] = static_cast<uint16_t>(rg);
          ncand += __popc(m);
        }
      }
    }
    if (ncand == 0) continue;
    __syncwarp();
    const bool every = ncand > kCandMax;  // list overflowed: scan every receptor residue
    const int nscan = every ? p.GR : ncand;
    const int A0 = p.lg_off[lg0], A1 = p.lg_off[lg1];
    const bool whole = A1 - A0 <= kUnitAtoms;
    bool moved = false;
    int nn = 0;
    // tests the listed residue pairs; base: first atom of s_f
    auto test = [&](int base) {
      __syncwarp();
      for (int q = 0; q < nn; q += 2) {
        bool on = q + half < nn;
        const uint32_t e = s_near[wib][on ? q + half : q];
        const int r = static_cast<int>(e & 0xffffu), i = static_cast<int>(e >> 16), lg = lg0 + i;
        const int b0 = p.rg_off[r], nb = p.rg_off[r + 1] - b0;
        const int a0 = p.lg_off[lg], na = p.lg_off[lg + 1] - a0;
        const float4 *laf = s_f[wib] + (a0 - base);
        const float4 ls = s_ls[wib][i];
        bool found = false;
        const bool big = on && (nb > 16 || na > 16);
        if (__any_sync(kFull, big)) {
          // a residue of more than 16 heavy atoms: the whole warp, one pair
          // after the other
          for (int s = 0; s < 2; ++s) {
            if (!__shfl_sync(kFull, big, 16 * s)) continue;
            const int B0 = __shfl_sync(kFull, b0, 16 * s), NB = __shfl_sync(kFull, nb, 16 * s),
                      S0 = __shfl_sync(kFull, a0, 16 * s), NA = __shfl_sync(kFull, na, 16 * s);
            bool hit = false;
            for (int b = B0; b < B0 + NB && !__any_sync(kFull, hit); ++b) {
              const float4 rb = p.r32[b];
              for (int a = lane; a < NA; a += 32) {
                const float4 la = s_f[wib][GD_DCHECK(p.err, S0 - base + a < kUnitAtoms, 30) ? S0 - base + a : 0];
                const float d2 = d2f(rb, la.x, la.y, la.z);
                if (d2 <= p.t32 + p.guard) hit = hit || d2 < p.t32 - p.guard || exact_contact(p, pose, b, S0 + a);
              }
            }
            const bool any = __any_sync(kFull, hit);
            if (half == s) found = any;
          }
        }
        on = on && !big;
        float4 ra = make_float4(0.0f, 0.0f, 0.0f, 0.0f), la = ra;
        bool cand = false;
        if (on && l16 < nb) {
          ra = p.r32[b0 + l16];
          const float dx = ra.x - ls.x, dy = ra.y - ls.y, dz = ra.z - ls.z, lim = ls.w + p.reach;
          cand = dx * dx + dy * dy + dz * dz <= lim * lim;
        }
        const bool atom = on && l16 < na;
        if (atom) la = laf[GD_DCHECK(p.err, laf + l16 < s_f[wib] + kUnitAtoms, 30) ? l16 : 0];
        unsigned m = (__ballot_sync(kFull, cand) >> (16 * half)) & 0xffffu;
        while (__any_sync(kFull, m != 0)) {
          const int j = m ? __ffs(m) - 1 : 0;
          const float bx = __shfl_sync(kFull, ra.x, 16 * half + j), by = __shfl_sync(kFull, ra.y, 16 * half + j),
                      bz = __shfl_sync(kFull, ra.z, 16 * half + j);
          bool hit = false;
          if (m && atom) {
            const float d2 = d2f(make_float4(bx, by, bz, 0.0f), la.x, la.y, la.z);
            if (d2 <= p.t32 + p.guard) hit = d2 < p.t32 - p.guard || exact_contact(p, pose, b0 + j, a0 + l16);
          }
          const unsigned h = (__ballot_sync(kFull, hit) >> (16 * half)) & 0xffffu;
          if (h) {
            found = true;
            m = 0;
          } else {
            m &= m - 1;
          }
        }
        const unsigned fm = __ballot_sync(kFull, found && l16 == 0);
        if (found && l16 == 0) s_out[wib][nout + (half && (fm & 1u) ? 1 : 0)] = static_cast<uint32_t>(r) * p.GL + lg;
        nout += __popc(fm);
        if (nout > kOutMax - 2) flush();
      }
      nn = 0;
      __syncwarp();
    };
    auto move_atoms = [&](int from, int to) {
      for (int a = from + lane; a < to; a += 32) s_f[wib][a - from] = move(p.l_rel[a]);
    };
    for (int lg = lg0; lg < lg1; ++lg) {
      const float4 ls = s_ls[wib][lg - lg0];
      const uint8_t lchain = p.lg_chain[lg];
      for (int k0 = 0; k0 < nscan; k0 += 32) {
        // 32 candidates at a time: the sphere test on one lane each
        const int k = k0 + lane;
        int rg = 0;
        bool near = false;
        if (k < nscan) {
          rg = every ? k : s_cand[wib][k];
          near = p.rg_chain[rg] != lchain && within(p.rg_sph[rg], ls);
        }
        const unsigned m = __ballot_sync(kFull, near);
        if (near) s_near[wib][nn + __popc(m & lt_mask)] = static_cast<uint32_t>(rg) | static_cast<uint32_t>(lg - lg0) << 16;
        nn += __popc(m);
        if (nn >= kNearMax || (!whole && k0 + 32 >= nscan && nn > 0)) {
          if (whole) {
            if (!moved) move_atoms(A0, A1);
            moved = true;
            test(A0);
          } else {
            const int a0 = p.lg_off[lg];
            move_atoms(a0, p.lg_off[lg + 1]);
            test(a0);
          }
        }
      }
    }
    if (nn > 0) {  // (whole units only: the others test after each residue)
      if (!moved) move_atoms(A0, A1);
      test(A0);
    }
    __syncwarp();
  }
  if (nout > 0) flush();
}

// Exclusive prefix sums (one CTA): of the set bits of a bitmap's words, or of
// counts; *total receives the sum.  With counts2 given, *max2 receives the
// largest of its n2 entries, and host_info (pinned) both.
template <bool BITS>
__global__ void __launch_bounds__(1024) k_scan(const uint32_t *v, long long words, int *base, int *total,
                                               const int *counts2, int n2, int *max2, int *host_info) {
  __shared__ int s_w[32];
  __shared__ int s_run;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int run = 0;
  // four consecutive words per thread and round; the next round's are loaded
  // before this one's sums meet
  auto load = [&](long long w) {
    uint4 x = make_uint4(0, 0, 0, 0);
    if (w + 3 < words) x = *reinterpret_cast<const uint4 *>(v + w);
    else {
      if (w < words) x.x = v[w];
      if (w + 1 < words) x.y = v[w + 1];
      if (w + 2 < words) x.z = v[w + 2];
    }
    if (BITS) x = make_uint4(__popc(x.x), __popc(x.y), __popc(x.z), __popc(x.w));
    return x;
  };
  uint4 next = load(4LL * t);
  for (long long w0 = 0; w0 < words; w0 += 4096) {
    const uint4 x = next;
    const long long w = w0 + 4LL * t;
    next = load(w + 4096);
    const int mine = static_cast<int>(x.x + x.y + x.z + x.w);
    int inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) s_w[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      const int own = s_w[lane];
      int sum = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, sum, o);
        if (lane >= o) sum += y;
      }
      s_w[lane] = sum - own;
      if (lane == 31) s_run = sum;
    }
    __syncthreads();
    int b = run + s_w[warp] + inc - mine;
    const int add[4] = {static_cast<int>(x.x), static_cast<int>(x.y), static_cast<int>(x.z), static_cast<int>(x.w)};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (w + k < words) base[w + k] = b;
      b += add[k];
    }
    run += s_run;
    __syncthreads();
  }
  if (t == 0) {
    *total = run;
    if (host_info) host_info[0] = run;
  }
  if (counts2) {
    int m = 0;
    for (int k = t; k < n2; k += 1024) m = max(m, counts2[k]);
    m = __reduce_max_sync(kFull, m);
    if (lane == 0) s_w[warp] = m;
    __syncthreads();
    if (warp == 0) {
      m = __reduce_max_sync(kFull, s_w[lane]);
      if (lane == 0) {
        *max2 = m;
        host_info[1] = m;
      }
    }
  }
}

// A contact's index in the compacted universe.
__device__ __forceinline__ int universe_index(const uint32_t *ubits, const int *base, uint32_t v) {
  return base[v >> 5] + __popc(ubits[v >> 5] & ((1u << (v & 31)) - 1u));
}

// The poses' lists as bitset rows over the compacted universe, one CTA per
// pose; a row is put together in shared memory when it fits (in_smem), else
// in place (rows cleared beforehand).
constexpr int kRowSmem = 4096;  // 64-bit words
__global__ void __launch_bounds__(256) k_rows(const uint32_t *lists, const int *counts, int cap, const uint32_t *ubits,
                                              const int *base, const int *info, int stride, int in_smem,
                                              unsigned long long *rows) {
  extern __shared__ uint32_t s_row[];
  const int pose = blockIdx.x, W = (info[0] + 63) / 64, c = min(counts[pose], cap);
  uint32_t *row = in_smem ? s_row : reinterpret_cast<uint32_t *>(rows + static_cast<size_t>(pose) * stride);
  if (in_smem) {
    for (int w = threadIdx.x; w < 2 * W; w += blockDim.x) s_row[w] = 0;
    __syncthreads();
  }
  for (int k = threadIdx.x; k < c; k += blockDim.x) {
    const int at = universe_index(ubits, base, lists[static_cast<size_t>(pose) * cap + k]);
    atomicOr(&row[at >> 5], 1u << (at & 31));
  }
  if (in_smem) {
    __syncthreads();
    uint32_t *out = reinterpret_cast<uint32_t *>(rows + static_cast<size_t>(pose) * stride);
    for (int w = threadIdx.x; w < 2 * W; w += blockDim.x) out[w] = s_row[w];
  }
}

// ---- FCC pair counts from per-contact pose lists ("postings") ----
// For poses whose contacts are spread (few poses per contact), the common
// count of a pose pair is the number of contacts whose list holds both: the
// work is the sum over contacts of k (k - 1) / 2 for k poses per contact,
// against n^2 / 2 pose pairs x W words for the bitsets.  Counts are exact
// integers either way, so the clusters are identical.

// Per contact (compacted index): how many poses make it.
__global__ void __launch_bounds__(256) k_post_count(const uint32_t *lists, const int *counts, int cap,
                                                    const uint32_t *ubits, const int *base, int n, int *kc) {
  for (int pose = blockIdx.x; pose < n; pose += gridDim.x) {
    const int c = min(counts[pose], cap);
    for (int k = threadIdx.x; k < c; k += blockDim.x)
      atomicAdd(&kc[universe_index(ubits, base, lists[static_cast<size_t>(pose) * cap + k])], 1);
  }
}

// Sum over contacts of k (k - 1) / 2: the pair increments of the posting path.
__global__ void k_post_work(const int *kc, int U, unsigned long long *sum) {
  unsigned long long acc = 0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < U; c += gridDim.x * blockDim.x) {
    const unsigned long long k = static_cast<unsigned long long>(kc[c]);
    acc += k * (k - (k > 0 ? 1 : 0)) / 2;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd(sum, acc);
}

// The poses of each contact, at offs[c] onwards (order within a list is
// free: the counts do not depend on it).
__global__ void __launch_bounds__(256) k_post_fill(const uint32_t *lists, const int *counts, int cap,
                                                   const uint32_t *ubits, const int *base, int n, const int *offs,
                                                   int *cursor, int *post) {
  for (int pose = blockIdx.x; pose < n; pose += gridDim.x) {
    const int c = min(counts[pose], cap);
    for (int k = threadIdx.x; k < c; k += blockDim.x) {
      const int at = universe_index(ubits, base, lists[static_cast<size_t>(pose) * cap + k]);
      post[offs[at] + atomicAdd(&cursor[at], 1)] = pose;
    }
  }
}

// One warp per contact: +1 on the common count of every pose pair in its list.
__global__ void k_post_pairs(const int *offs, const int *kc, const int *post, int U, int n, uint32_t *common) {
  const int lane = threadIdx.x & 31;
  for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < U; c += (gridDim.x * blockDim.x) >> 5) {
    const int k = kc[c], o = offs[c];
    for (int a = 0; a + 1 < k; ++a) {
      const int i = post[o + a];
      for (int b = a + 1 + lane; b < k; b += 32) {
        const int j = post[o + b];
        const int lo = min(i, j), hi = max(i, j);
        atomicAdd(&common[static_cast<size_t>(lo) * n + hi], 1u);
      }
    }
  }
}

// The edges from the common counts of the pairs i <= j (the diagonal: the
// pose's own size), as k_fcc decides them.
__global__ void k_post_decide(const uint32_t *common, const int *sizes, int n, double c, double cs, uint32_t *adj,
                              int adj_words, int c0) {
  const float c32 = static_cast<float>(c), cs32 = static_cast<float>(cs);
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int si = sizes[i] + c0;
    for (int j = i + threadIdx.x; j < n; j += blockDim.x) {
      const int e = fcc_edges(i == j ? si : static_cast<int>(common[static_cast<size_t>(i) * n + j]) + c0, si,
                              sizes[j] + c0, c, cs, c32, cs32);
      if (e & 1) atomicOr(&adj[static_cast<size_t>(i) * adj_words + (j >> 5)], 1u << (j & 31));
      if ((e & 2) && j != i) atomicOr(&adj[static_cast<size_t>(j) * adj_words + (i >> 5)], 1u << (i & 31));
    }
  }
}

// ---- greedy clustering ----

// cluster_elements (src/clustering.rs:183-254) over the adjacency bit matrix
// (row e, bit m: edge e -> m), by one CTA, or one cluster of kGreedyCtas CTAs
// that split the rows:
//  - count[e] = unused neighbours of e (its self-edge included, as in the
//    reference); the centre is the unused element with the largest count,
//    lower index on ties (each CTA's best through the others' shared memory).
//  - A cluster M holds the centre and its unused neighbours, so its size is at
//    most count + 1 (+1 only without a self-edge, i.e. an empty contact set).
//    Counts never grow, so once the best count + 1 is below min_size every
//    later cluster would be dropped by the size filter: the loop stops there
//    without changing the kept clusters or their order.
//  - An edge of any element implies its self-edge (a ratio never exceeds 1), so
//    once the best count is 1, every element left is alone in its cluster, those
//    with a self-edge first, each in index order.  The loop stops there too: where
//    such clusters are kept (min_size <= 1) the host numbers them.  (880 poses
//    without a common contact: 2.3 ms with a round each.)
//  - After a cluster is formed, every unused e loses |N(e) & M|.
// Every CTA keeps the used and member bits of all elements and derives the
// same cluster; label[e] receives its number, centers[k] the centres.
// On the host the counting of 4,096 poses' rows took 2.75 ms (0.15 here).
constexpr int kGreedyCtas = 8;         // at most; one CTA where the matrix fits its shared memory
constexpr int kGreedyThreads = 1024;
constexpr size_t kGreedyAdj = 96 * 1024;  // bytes of such a matrix
constexpr int kGreedyMax = 65536;  // elements (shared memory); beyond: the host
struct GreedySmem {
  size_t used, memb, nz, count, adj, total;
};
__host__ __device__ inline bool greedy_alone(int n) {
  return static_cast<size_t>(n) * ((static_cast<size_t>(n) + 31) / 32) * 4 <= kGreedyAdj;
}
__host__ __device__ inline GreedySmem greedy_smem(int n) {
  GreedySmem L;
  const size_t words = (static_cast<size_t>(n) + 31) / 32, ctas = greedy_alone(n) ? 1 : kGreedyCtas,
               rows = (static_cast<size_t>(n) + ctas - 1) / ctas;
  size_t o = 0;
  L.used = o;
  o += 4 * words;
  L.memb = o;
  o += 4 * words;
  L.nz = o;  // the words with members
  o += 4 * words;
  L.count = o;  // -1: used
  o += 4 * rows;
  L.adj = o;
  if (greedy_alone(n)) o += 4 * words * rows;
  L.total = (o + 15) / 16 * 16;
  return L;
}
__global__ void __launch_bounds__(kGreedyThreads)
    k_greedy(const uint32_t *g_adj, int n, int words, int min_size, int *label, int *centers, int *n_clusters) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int2 s_best[2][kGreedyCtas], s_warp[kGreedyThreads / 32];
  __shared__ int s_nnz;
  const GreedySmem L = greedy_smem(n);
  uint32_t *used = reinterpret_cast<uint32_t *>(smem + L.used), *memb = reinterpret_cast<uint32_t *>(smem + L.memb);
  int *nz = reinterpret_cast<int *>(smem + L.nz), *count = reinterpret_cast<int *>(smem + L.count);
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank()), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nt = blockDim.x, kW = nt >> 5;
  const int nc = static_cast<int>(cluster.num_blocks()), per = (n + nc - 1) / nc, e0 = min(n, rank * per), e1 = min(n, e0 + per), rows = e1 - e0;
  const uint32_t *adj = g_adj;
  if (nc == 1 && greedy_alone(n)) {
    uint32_t *s_adj = reinterpret_cast<uint32_t *>(smem + L.adj);
    for (int i = tid; i < n * words; i += nt) s_adj[i] = g_adj[i];
    adj = s_adj;
    __syncthreads();
  }
  for (int w = tid; w < words; w += nt) used[w] = 0;
  for (int r = warp; r < rows; r += kW) {
    const uint32_t *row = adj + static_cast<size_t>(e0 + r) * words;
    int c = 0;
    for (int w = lane; w < words; w += 32) c += __popc(row[w]);
    c = __reduce_add_sync(kFull, c);
    if (lane == 0) {
      count[r] = c;
      label[e0 + r] = -1;
    }
  }
  // (every CTA has started before its s_best is written to)
  if (nc > 1) cluster.sync();
  else __syncthreads();
  int k = 0;
  for (;; ++k) {
    // the unused element with the largest count, lower index on ties: the
    // count + 1 and the index of each warp's, CTA's and the cluster's best
    int top = 0, at = 0x7fffffff;
    for (int r = tid; r < rows; r += nt)
      if (count[r] + 1 > top) {
        top = count[r] + 1;
        at = e0 + r;
      }
    const int wtop = __reduce_max_sync(kFull, top);
    const int wat = __reduce_min_sync(kFull, top == wtop ? at : 0x7fffffff);
    if (lane == 0) s_warp[warp] = make_int2(wtop, wat);
    __syncthreads();
    if (warp == 0) {
      const int2 w = lane < kW ? s_warp[lane] : make_int2(0, 0x7fffffff);
      const int ctop = __reduce_max_sync(kFull, w.x), cat = __reduce_min_sync(kFull, w.x == ctop ? w.y : 0x7fffffff);
      if (lane < nc) *(nc > 1 ? cluster.map_shared_rank(&s_best[k & 1][rank], lane) : &s_best[k & 1][0]) = make_int2(ctop, cat);
    }
    if (tid == 0) s_nnz = 0;
    if (nc > 1) cluster.sync();  // (two slots: the next round's writes cannot meet this one's reads)
    else __syncthreads();
    int2 best = s_best[k & 1][0];
    for (int c = 1; c < nc; ++c)  // (the CTAs' rows ascend: the first of equals has the lower index)
      if (s_best[k & 1][c].x > best.x) best = s_best[k & 1][c];
    if (best.x < max(min_size, 3)) break;  // best count + 1 < min_size, or none left but clusters of one
    const int center = best.y;
    // the members: the centre's unused neighbours and the centre
    const uint32_t *crow = adj + static_cast<size_t>(center) * words;
    for (int w = tid; w < words; w += nt) {
      uint32_t m = crow[w] & ~used[w];
      if (w == (center >> 5)) m |= 1u << (center & 31);
      memb[w] = m;
      used[w] |= m;
      if (m) nz[atomicAdd(&s_nnz, 1)] = w;
    }
    if (rank == 0 && tid == 0) centers[k] = center;
    __syncthreads();
    const int nnz = s_nnz;
    // members are used up, the others lose their edges into the cluster
    auto settle = [&](int r, int lost) {
      const int e = e0 + r;
      if ((memb[e >> 5] >> (e & 31)) & 1u) {
        count[r] = -1;
        label[e] = k;
      } else if (count[r] >= 0) {
        count[r] -= lost;
      }
    };
    if (nnz >= 8) {
      // four rows of a warp and four of their words per lane at a time, to
      // have sixteen loads in flight
      for (int r0 = warp; r0 < rows; r0 += 4 * kW) {
        int c[4] = {0, 0, 0, 0};
        for (int i0 = lane; i0 < nnz; i0 += 128) {
          uint32_t v[4][4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = i0 + 32 * q, w = i < nnz ? nz[i] : 0;
            const uint32_t m = i < nnz ? memb[w] : 0u;
#pragma unroll
            for (int u = 0; u < 4; ++u)
              v[q][u] = adj[static_cast<size_t>(e0 + min(r0 + u * kW, rows - 1)) * words + w] & m;
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int u = 0; u < 4; ++u) c[u] += __popc(v[q][u]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int t = __reduce_add_sync(kFull, c[u]);
          if (lane == 0 && r0 + u * kW < rows) settle(r0 + u * kW, t);
        }
      }
    } else {  // few words: a thread per row
      for (int r = tid; r < rows; r += nt) {
        const uint32_t *row = adj + static_cast<size_t>(e0 + r) * words;
        int c = 0;
        for (int i = 0; i < nnz; ++i) c += __popc(row[nz[i]] & memb[nz[i]]);
        settle(r, c);
      }
    }
    __syncthreads();
  }
  if (rank == 0 && tid == 0) *n_clusters = k;
  if (min_size <= 1)
    for (int r = tid; r < rows; r += nt)
      if (count[r] == 0) label[e0 + r] = -2;  // left, and without a self-edge
  if (nc > 1) cluster.sync();  // nobody leaves while its slots are being written
}

// host mirror of the device transform (same operation order, no fused ops)
void xform_host(const gd_pose_frame &f, double cx, double cy, double cz, double xo, double yo, double zo, double &X,
                double &Y, double &Z) {
  const double x = xo - cx, y = yo - cy, z = zo - cz;
  const double nx = x * f.ca * f.cb + y * f.m01 + z * f.m02;
  const double ny = x * f.sa * f.cb + y * f.m11 + z * f.m12;
  const double nz = -x * f.sb + y * f.cb * f.sg + z * f.cb * f.cg;
  X = nx + cx + f.dx;
  Y = ny + cy + f.dy;
  Z = nz + cz + f.dz;
}

inline int64_t canon(int64_t ka, int64_t kb) {
  // "cA rA cB rB" with the smaller chain first (src/clustering.rs:100-105)
  const int64_t ca = ka >> 16, cb = kb >> 16;
  if (ca > cb) std::swap(ka, kb);
  return ((ka >> 16) << 48) | ((ka & 0xffff) << 32) | ((kb >> 16) << 16) | (kb & 0xffff);
}

// Inter-chain contacts among the residues of one molecule at coordinates x,
// y, z (host; multi-chain receptors once, multi-chain ligands per pose):
// residue pairs on different chains with an atom pair at d2 <= t_le.  Pairs
// whose enclosing spheres are beyond the cutoff are skipped.  When unstable is
// given it is set if some residue pair's closest atom pair lies within a
// relative 1e-6 of t_le: a decision that the FP64 rounding of a rigid
// transform (some 1e-12 A^2 on d2) could not flip lies far outside that.
void intra_contacts(const std::vector<int64_t> &gkey, const std::vector<int> &goff, const std::vector<int> &atoms,
                    const double *x, const double *y, const double *z, double t_le, std::vector<int64_t> &out,
                    bool *unstable = nullptr) {
  const int G = static_cast<int>(gkey.size());
  std::vector<double> c(3 * static_cast<size_t>(G)), r(G);
  for (int g = 0; g < G; ++g)
    enclosing_ball(x, y, z, atoms.data() + goff[g], goff[g + 1] - goff[g], &c[3 * static_cast<size_t>(g)], r[g]);
  // a skipped pair's closest atoms lie beyond the cutoff by more than the band
  const double band = 1e-6 * t_le, reach = std::sqrt(t_le) + 1e-4;
  for (int g = 0; g < G; ++g)
    for (int h = g + 1; h < G; ++h) {
      if ((gkey[g] >> 16) == (gkey[h] >> 16)) continue;
      const double *cg = &c[3 * static_cast<size_t>(g)], *ch = &c[3 * static_cast<size_t>(h)];
      const double ex = cg[0] - ch[0], ey = cg[1] - ch[1], ez = cg[2] - ch[2];
      const double lim = r[g] + r[h] + reach;
      if (ex * ex + ey * ey + ez * ez > lim * lim * (1.0 + 1e-9)) continue;
      double best = INFINITY;
      for (int a = goff[g]; a < goff[g + 1] && !(best < t_le - band); ++a)
        for (int b = goff[h]; b < goff[h + 1]; ++b) {
          const int ia = atoms[a], ib = atoms[b];
          const double dx = x[ia] - x[ib], dy = y[ia] - y[ib], dz = z[ia] - z[ib];
          best = std::min(best, dx * dx + dy * dy + dz * dz);
          if (best < t_le - band) break;
        }
      if (best <= t_le) out.push_back(canon(gkey[g], gkey[h]));
      if (unstable && std::fabs(best - t_le) <= band) *unstable = true;
    }
}

// The topology's device arrays, staged on the host and copied in one piece
// (each 256-byte aligned): one cudaMalloc and one cudaMemcpy per complex.
struct TopoPack {
  struct Item {
    const void *src;
    size_t bytes, off;
    std::function<void(char *)> bind;
  };
  std::vector<Item> items;
  size_t total = 0;
  template <typename T>
  void add(const std::vector<T> &h, T **d) {
    const size_t off = total;
    items.push_back(Item{h.empty() ? nullptr : h.data(), sizeof(T) * h.size(), off,
                         [d, off](char *base) { *d = reinterpret_cast<T *>(base + off); }});
    total += (sizeof(T) * std::max<size_t>(h.size(), 1) + 255) / 256 * 256;
  }
  gd_status commit(gd_context *ctx, ClusterTopo *t) {
    void *p = nullptr;
    gd_status s = dev_alloc(ctx, total, &p);
    if (s != GD_OK) return s;
    t->allocs.push_back(p);
    t->bytes += total;
    std::vector<char> h(total, 0);
    for (const Item &it : items)
      if (it.bytes) std::memcpy(h.data() + it.off, it.src, it.bytes);
    const cudaError_t e = cudaMemcpy(p, h.data(), total, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaMemcpy (contact topology)");
    for (const Item &it : items) it.bind(static_cast<char *>(p));
    return GD_OK;
  }
};

void group_atoms(const std::vector<uint8_t> &chain, const std::vector<int16_t> &res, const std::vector<uint8_t> &elem,
                 std::vector<int64_t> &gkey, std::vector<int> &goff, std::vector<int> &atoms) {
  std::map<int64_t, std::vector<int>> g;
  int64_t last = -1;
  std::vector<int> *at = nullptr;  // the last atom's residue (usually the next one's too)
  for (size_t i = 0; i < chain.size(); ++i) {
    if (elem[i] == GD_ELEM_H) continue;  // src/clustering.rs:67-70
    const int64_t key = (static_cast<int64_t>(chain[i]) << 16) | static_cast<uint16_t>(res[i]);
    if (key != last) at = &g[last = key];
    at->push_back(static_cast<int>(i));
  }
  goff.assign(1, 0);
  for (auto &kv : g) {
    gkey.push_back(kv.first);
    atoms.insert(atoms.end(), kv.second.begin(), kv.second.end());
    goff.push_back(static_cast<int>(atoms.size()));
  }
}

// Residue groups put into spatially compact runs of `unit` (and, within, of
// `sub`) by their centroids, so that a block of consecutive groups has a small
// enclosing sphere whatever the chain's course.  Returns each group's index before
// (by key: its rank).
std::vector<int> compact_groups(const std::vector<double> &x, const std::vector<double> &y, const std::vector<double> &z,
                                std::vector<int64_t> &gkey, std::vector<int> &goff, std::vector<int> &atoms, int unit,
                                int sub) {
  const int G = static_cast<int>(gkey.size());
  std::vector<double> c[3];
  for (int g = 0; g < G; ++g) {
    double m[3] = {0.0, 0.0, 0.0};
    for (int a = goff[g]; a < goff[g + 1]; ++a) {
      m[0] += x[atoms[a]];
      m[1] += y[atoms[a]];
      m[2] += z[atoms[a]];
    }
    for (int k = 0; k < 3; ++k) c[k].push_back(m[k] / (goff[g + 1] - goff[g]));
  }
  const std::vector<int> order = compact_runs(c[0].data(), c[1].data(), c[2].data(), G, unit, sub);
  std::vector<int64_t> key;
  std::vector<int> off{0}, at;
  for (int g : order) {
    key.push_back(gkey[g]);
    at.insert(at.end(), atoms.begin() + goff[g], atoms.begin() + goff[g + 1]);
    off.push_back(static_cast<int>(at.size()));
  }
  gkey.swap(key);
  goff.swap(off);
  atoms.swap(at);
  return order;
}

gd_status build_topo(gd_complex *cx, ClusterTopo **out) {
  gd_context *ctx = cx->ctx;
  ClusterTopo *t = new ClusterTopo();
  group_atoms(cx->h_rchain, cx->h_rres, cx->h_relem, t->rg_key, t->rg_off, t->r_atoms);
  group_atoms(cx->h_lchain, cx->h_lres, cx->h_lelem, t->lg_key, t->lg_off, t->l_atoms);
  t->GR = static_cast<int>(t->rg_key.size());
  t->GL = static_cast<int>(t->lg_key.size());
  for (int g = 1; g < t->GR; ++g) t->multi_chain_rec |= (t->rg_key[g] >> 16) != (t->rg_key[0] >> 16);
  for (int g = 1; g < t->GL; ++g) t->multi_chain_lig |= (t->lg_key[g] >> 16) != (t->lg_key[0] >> 16);
  {
    std::vector<int64_t> a = t->rg_key, b = t->lg_key, both;
    std::set_intersection(a.begin(), a.end(), b.begin(), b.end(), std::back_inserter(both));
    t->mixed = !both.empty();
  }
  if (t->multi_chain_rec) t->r_by_key = {t->rg_key, t->rg_off, t->r_atoms};
  if (t->multi_chain_lig) t->l_by_key = {t->lg_key, t->lg_off, t->l_atoms};
  t->rg_rank = compact_groups(cx->h_rx, cx->h_ry, cx->h_rz, t->rg_key, t->rg_off, t->r_atoms, 32, 8);
  t->lg_rank = compact_groups(cx->h_lx, cx->h_ly, cx->h_lz, t->lg_key, t->lg_off, t->l_atoms, kLigBlock, kLigBlock / 4);
  std::vector<double> rx, ry, rz, lx, ly, lz;
  for (int i : t->r_atoms) {
    rx.push_back(cx->h_rx[i]);
    ry.push_back(cx->h_ry[i]);
    rz.push_back(cx->h_rz[i]);
  }
  for (int i : t->l_atoms) {
    lx.push_back(cx->h_lx[i]);
    ly.push_back(cx->h_ly[i]);
    lz.push_back(cx->h_lz[i]);
  }
  std::vector<float4> r32(rx.size());
  for (size_t a = 0; a < rx.size(); ++a)
    r32[a] = make_float4(static_cast<float>(rx[a] - cx->ox), static_cast<float>(ry[a] - cx->oy),
                         static_cast<float>(rz[a] - cx->oz), 0.0f);
  // Spheres enclosing the atoms of every residue, of blocks of kLigBlock
  // consecutive ligand residues and of 32 receptor residues (each slightly
  // widened), on the host pool: sixteen passes over every atom for each kind,
  // half of a first call on a large complex when they ran on one thread.
  const int nb = (t->GL + kLigBlock - 1) / kLigBlock, nrb = (t->GR + 31) / 32;
  std::vector<float4> rsph(t->GR), rbsph(std::max(nrb, 1), make_float4(0, 0, 0, 0));
  std::vector<D4> lsph(t->GL), lbsph(std::max(nb, 1), D4{0, 0, 0, 0});
  std::vector<uint8_t> rch(t->GR), lch(t->GL);
  for (int g = 0; g < t->GR; ++g) rch[g] = static_cast<uint8_t>(t->rg_key[g] >> 16);
  for (int g = 0; g < t->GL; ++g) lch[g] = static_cast<uint8_t>(t->lg_key[g] >> 16);
  auto ball = [](const std::vector<double> &x, const std::vector<double> &y, const std::vector<double> &z, int a0, int a1) {
    double c[3], r;
    enclosing_ball(x.data() + a0, y.data() + a0, z.data() + a0, nullptr, a1 - a0, c, r);
    return D4{c[0], c[1], c[2], r * (1 + 1e-6) + 1e-3};
  };
  auto rec_ball = [&](int g0, int g1) {
    const D4 v = ball(rx, ry, rz, t->rg_off[g0], t->rg_off[g1]);
    return make_float4(static_cast<float>(v.x - cx->ox), static_cast<float>(v.y - cx->oy), static_cast<float>(v.z - cx->oz),
                       static_cast<float>(v.w));
  };
  const int nt = rx.size() + lx.size() >= 2048 ? 32 : 1;
  auto spheres = [&](int task) {
    auto each = [&](int n, auto f) {
      for (int i = static_cast<int>(static_cast<long long>(n) * task / nt); i < static_cast<long long>(n) * (task + 1) / nt; ++i) f(i);
    };
    each(t->GR, [&](int g) { rsph[g] = rec_ball(g, g + 1); });
    each(nrb, [&](int b) { rbsph[b] = rec_ball(b * 32, std::min(t->GR, b * 32 + 32)); });
    each(t->GL, [&](int g) { lsph[g] = ball(lx, ly, lz, t->lg_off[g], t->lg_off[g + 1]); });
    each(nb, [&](int b) {
      lbsph[b] = ball(lx, ly, lz, t->lg_off[b * kLigBlock], t->lg_off[std::min(t->GL, (b + 1) * kLigBlock)]);
    });
  };
  if (nt == 1) spheres(0);
  else host_parallel(nt, spheres);
  // the same relative to the rotation centre, as the contact kernel moves them
  auto rel = [&](const D4 &v) { return D4{v.x - cx->cx, v.y - cx->cy, v.z - cx->cz, v.w}; };
  auto rel32 = [&](const D4 &v) {
    const D4 r = rel(v);
    return make_float4(static_cast<float>(r.x), static_cast<float>(r.y), static_cast<float>(r.z), static_cast<float>(r.w));
  };
  std::vector<float4> lgrel(t->GL), lbrel(std::max(nb, 1), make_float4(0, 0, 0, 0));
  std::vector<D4> lrel(lx.size());
  for (int g = 0; g < t->GL; ++g) lgrel[g] = rel32(lsph[g]);
  for (int b = 0; b < nb; ++b) lbrel[b] = rel32(lbsph[b]);
  for (size_t a = 0; a < lx.size(); ++a) lrel[a] = rel(D4{lx[a], ly[a], lz[a], 0.0});
  // one allocation and one copy for every array of the topology
  TopoPack pack;
  pack.add(rbsph, &t->d_rb_sph);
  pack.add(lgrel, &t->d_lg_rel);
  pack.add(lbrel, &t->d_lb_rel);
  pack.add(lrel, &t->d_l_rel);
  pack.add(rx, &t->d_rx);
  pack.add(ry, &t->d_ry);
  pack.add(rz, &t->d_rz);
  pack.add(lx, &t->d_lx);
  pack.add(ly, &t->d_ly);
  pack.add(lz, &t->d_lz);
  pack.add(t->rg_off, &t->d_rg_off);
  pack.add(t->lg_off, &t->d_lg_off);
  pack.add(rsph, &t->d_rg_sph);
  pack.add(lsph, &t->d_lg_sph);
  pack.add(rch, &t->d_rg_chain);
  pack.add(lch, &t->d_lg_chain);
  pack.add(r32, &t->d_r32);
  const gd_status s = pack.commit(ctx, t);
  if (s != GD_OK) {
    for (void *q : t->allocs) cudaFree(q);
    ctx->in_use -= std::min<uint64_t>(ctx->in_use, t->bytes);
    delete t;
    return s;
  }
  *out = t;
  return GD_OK;
}

gd_status get_topo(gd_complex *cx, ClusterTopo **t) {
  if (!cx->cluster_cache) {
    ClusterTopo *nt = nullptr;
    gd_status s = build_topo(cx, &nt);
    if (s != GD_OK) return s;
    cx->cluster_cache = nt;
  }
  *t = static_cast<ClusterTopo *>(cx->cluster_cache);
  return GD_OK;
}

// The clusters of at least min_size in gdock's output order (a stable sort by
// size, src/clustering.rs:289-292) from each element's cluster and the
// centres, both in the order the greedy pass formed them; members ascending.
int order_clusters(const int *label, const int *center, int k, int n, int min_size, int32_t *centers, int32_t *sizes,
                   int32_t *members) {
  std::vector<int> size(k, 0), order(k), at(k, -1);
  for (int e = 0; e < n; ++e)
    if (label[e] >= 0) ++size[label[e]];
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return size[a] > size[b]; });
  int kept = 0, mo = 0;
  for (int c : order) {
    if (size[c] < min_size) continue;
    centers[kept] = center[c];
    sizes[kept] = size[c];
    at[c] = mo;
    mo += size[c];
    ++kept;
  }
  for (int e = 0; e < n; ++e)
    if (label[e] >= 0 && at[label[e]] >= 0) members[at[label[e]]++] = e;
  return kept;
}

// The clusters of one that k_greedy leaves (labels -1, then -2), k clusters so
// far; returns the number of all.
int label_singles(int *label, int *center, int k, int n) {
  for (int kind : {-1, -2})
    for (int e = 0; e < n; ++e)
      if (label[e] == kind) {
        center[k] = e;
        label[e] = k++;
      }
  return k;
}

// k_greedy's clusters on the host, for more elements than it takes.
int greedy_labels(const std::vector<uint32_t> &adj, int n, int words, int min_size, std::vector<int> &label,
                  std::vector<int> &center) {
  std::vector<int> count(n, 0);
  for (int e = 0; e < n; ++e)
    for (int w = 0; w < words; ++w) count[e] += __builtin_popcount(adj[static_cast<size_t>(e) * words + w]);
  std::vector<uint32_t> used(words, 0), memb(words);
  label.assign(n, -1);
  center.clear();
  for (int k = 0;; ++k) {
    int best = -1, c = -1;
    for (int e = 0; e < n; ++e)
      if (label[e] < 0 && count[e] > best) {
        best = count[e];
        c = e;
      }
    if (c < 0 || best + 1 < min_size) return k;
    center.push_back(c);
    for (int w = 0; w < words; ++w) {
      memb[w] = adj[static_cast<size_t>(c) * words + w] & ~used[w];
      if (w == (c >> 5)) memb[w] |= 1u << (c & 31);
      used[w] |= memb[w];
      for (uint32_t v = memb[w]; v; v &= v - 1) label[w * 32 + __builtin_ctz(v)] = k;
    }
    for (int e = 0; e < n; ++e) {
      if (label[e] >= 0) continue;
      const uint32_t *row = &adj[static_cast<size_t>(e) * words];
      for (int w = 0; w < words; ++w)
        if (memb[w]) count[e] -= __builtin_popcount(row[w] & memb[w]);
    }
  }
}

size_t al256(size_t b) { return (b + 255) / 256 * 256; }

// Device bytes of a greedy pass's results: cluster count, labels, centres.
size_t greedy_bytes(int n) { return 256 + 2 * al256(sizeof(int) * static_cast<size_t>(n)); }

// Up to this many elements k_greedy writes its results, a word or two an
// element, to pinned memory itself.  With that, the universe's size written
// there by k_scan, one clearing pass instead of three and frames read in place,
// a call on 183 poses of 1,074 x 741 atoms went from 138 to 112 us (on 4,096 of
// 2,000 x 500 residues from 2,104 to 2,094).
constexpr int kGreedyDirect = 4096;

// Greedy clustering of the adjacency matrix d_adj (rows of `words`), its
// results through d_buf (greedy_bytes) into the caller's arrays; waits for the
// stream and reports device-side errors.
gd_status greedy_clusters(gd_context *ctx, const uint32_t *d_adj, int n, int words, int min_size, void *d_buf,
                          int32_t *n_clusters, int32_t *centers, int32_t *sizes, int32_t *members) {
  cudaStream_t st = ctx->stream;
  cudaError_t e = cudaSuccess;
  if (n > kGreedyMax) {
    std::vector<uint32_t> adj(static_cast<size_t>(n) * words);
    e = cudaMemcpyAsync(adj.data(), d_adj, sizeof(uint32_t) * adj.size(), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "FCC on the device");
    const gd_status s = check_device_error(ctx);
    if (s != GD_OK) return s;
    std::vector<int> label, center;
    const int k = greedy_labels(adj, n, words, min_size, label, center);
    *n_clusters = order_clusters(label.data(), center.data(), k, n, min_size, centers, sizes, members);
    return GD_OK;
  }
  char *b = static_cast<char *>(d_buf);
  const size_t lb = al256(sizeof(int) * static_cast<size_t>(n)), total = greedy_bytes(n);
  int *d_k = reinterpret_cast<int *>(b), *d_label = reinterpret_cast<int *>(b + 256),
      *d_center = reinterpret_cast<int *>(b + 256 + lb);
  gd_status s = ensure_scratch(ctx, 0, total);
  if (s != GD_OK) return s;
  char *h = static_cast<char *>(ctx->h_pinned);
  const bool direct = n <= kGreedyDirect;
  if (direct) {
    d_k = reinterpret_cast<int *>(h);
    d_label = reinterpret_cast<int *>(h + 256);
    d_center = reinterpret_cast<int *>(h + 256 + lb);
  }
  const size_t smem = greedy_smem(n).total;
  if (smem > 40 * 1024)
    e = cudaFuncSetAttribute(k_greedy, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e == cudaSuccess) {
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(greedy_alone(n) ? 1 : kGreedyCtas);
    // (a thread per row of a small matrix: fewer warps meet at the barriers)
    lc.blockDim = dim3(std::min(kGreedyThreads, std::max(128, (n + 31) / 32 * 32)));
    lc.dynamicSmemBytes = smem;
    lc.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = lc.gridDim.x;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    lc.attrs = &at;
    lc.numAttrs = 1;
    e = cudaLaunchKernelEx(&lc, k_greedy, d_adj, n, words, min_size, d_label, d_center, d_k);
  }
  if (e == cudaSuccess && !direct) e = cudaMemcpyAsync(h, b, total, cudaMemcpyDeviceToHost, st);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "greedy clustering");
  if ((s = finish_stream(ctx, st, "FCC on the device")) != GD_OK) return s;
  int *label = reinterpret_cast<int *>(h + 256), *center = reinterpret_cast<int *>(h + 256 + lb), k = *reinterpret_cast<int *>(h);
  if (min_size <= 1) k = label_singles(label, center, k, n);
  *n_clusters = order_clusters(label, center, k, n, min_size, centers, sizes, members);
  return GD_OK;
}

}  // namespace

void free_cluster_cache(gd_complex *cx) {
  if (!cx->cluster_cache) return;
  ClusterTopo *t = static_cast<ClusterTopo *>(cx->cluster_cache);
  for (void *p : t->allocs) cudaFree(p);
  cx->ctx->in_use -= std::min<uint64_t>(cx->ctx->in_use, t->bytes);
  delete t;
  cx->cluster_cache = nullptr;
}

// k_contacts serves receptors and ligands that share no residue, with ligand
// residues of at most kMaxGroupAtoms heavy atoms, entries that fit 32 bits and
// receptor residue numbers that fit 16; single-chain ones only unless
// multi_chain (clustering adds the inter-chain contacts within each molecule
// as a constant; per-pose contact lists take the other kernel for them).
bool fast_contacts_ok(const ClusterTopo *t, bool multi_chain = false) {
  if (t->mixed || (!multi_chain && (t->multi_chain_rec || t->multi_chain_lig))) return false;
  for (int g = 0; g < t->GL; ++g)
    if (t->lg_off[g + 1] - t->lg_off[g] > kMaxGroupAtoms) return false;
  return t->GR <= 65535 && static_cast<long long>(t->GR) * t->GL <= static_cast<long long>(UINT32_MAX);
}

// Words of the union bitmap over all (receptor residue, ligand residue) pairs.
long long pair_words(const ClusterTopo *t) {
  return std::max<long long>(1, (static_cast<long long>(t->GR) * t->GL + 31) / 32);
}

// List entries per pose (a pose with more makes the pass run again): 2,048
// cover docked poses of most complexes; large ones get up to 8,192, as many as
// a bit per residue pair would take (poses sunk into a receptor of 2,000
// residues pass 2,048, and the second pass took 8.5 ms of 22 for 4,096 poses).
// Fewer where the lists would pass 4 GiB or half of what a budget has left.
int list_cap(const gd_context *ctx, const ClusterTopo *t, int n) {
  const long long pairs = std::max<long long>(static_cast<long long>(t->GR) * t->GL, 1);
  long long cap = std::min(pairs, std::max(2048LL, std::min(8192LL, pairs / 32)));
  long long most = 4LL << 30;
  if (ctx->budget) {
    const uint64_t used = ctx->in_use - std::min<uint64_t>(ctx->in_use, ctx->d_scratch_bytes);
    most = std::min<long long>(most, static_cast<long long>(ctx->budget - std::min(ctx->budget, used)) / 2);
  }
  while (cap > 64 && cap * n * static_cast<long long>(sizeof(uint32_t)) > most) cap /= 2;
  return static_cast<int>(cap);
}

double max_displacement(const double *genes, int n) {
  double maxd = 0.0;
  for (int i = 0; i < n; ++i)
    for (int k = 3; k < 6; ++k) maxd = std::max(maxd, std::fabs(genes[6 * static_cast<size_t>(i) + k]));
  return maxd;
}

// Contact lists of n device-resident poses (d_counts is cleared; d_ubits, the
// union, too when given).  maxd bounds the poses' |displacement| components
// (it sizes the FP32 guard band, as for the scoring kernels).
gd_status launch_contacts(gd_complex *cx, ClusterTopo *t, const gd_pose_frame *d_frames, int n, double cutoff,
                          double maxd, int *d_counts, uint32_t *d_lists, int cap, uint32_t *d_ubits, cudaStream_t st,
                          uint32_t *d_rows = nullptr, long long row_words = 0) {
  gd_context *ctx = cx->ctx;
  // counts and union in one pass where the union follows the counts
  const size_t cb = al256(sizeof(int) * static_cast<size_t>(n)), ub = sizeof(uint32_t) * pair_words(t);
  const bool joined = d_ubits && reinterpret_cast<char *>(d_ubits) == reinterpret_cast<char *>(d_counts) + cb;
  cudaError_t e = cudaMemsetAsync(d_counts, 0, joined ? cb + ub : sizeof(int) * static_cast<size_t>(n), st);
  if (e == cudaSuccess && d_ubits && !joined) e = cudaMemsetAsync(d_ubits, 0, ub, st);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "contacts setup");
  if (t->GR == 0 || t->GL == 0 || n == 0) return GD_OK;
  ContactListParams p{};
  p.r32 = t->d_r32;
  p.rx = t->d_rx;
  p.ry = t->d_ry;
  p.rz = t->d_rz;
  p.rg_off = t->d_rg_off;
  p.rg_sph = t->d_rg_sph;
  p.rb_sph = t->d_rb_sph;
  p.rg_chain = t->d_rg_chain;
  p.lx = t->d_lx;
  p.ly = t->d_ly;
  p.lz = t->d_lz;
  p.lg_off = t->d_lg_off;
  p.l_rel = t->d_l_rel;
  p.lg_rel = t->d_lg_rel;
  p.lb_rel = t->d_lb_rel;
  p.lg_chain = t->d_lg_chain;
  p.GR = t->GR;
  p.GL = t->GL;
  p.cx = cx->cx;
  p.cy = cx->cy;
  p.cz = cx->cz;
  p.ox = cx->ox;
  p.oy = cx->oy;
  p.oz = cx->oz;
  p.frames = d_frames;
  p.t_le = make_thresholds(cutoff).contact_le;
  p.t32 = static_cast<float>(p.t_le);
  {
    // FP32 error bound of d2 near the cutoff (as for the scoring guard bands)
    const double u = std::ldexp(1.0, -24), c = cutoff;
    const double M = std::max(cx->rec_extent, cx->lig_radius + maxd +
                                                  std::max({std::fabs(cx->cx - cx->ox), std::fabs(cx->cy - cx->oy),
                                                            std::fabs(cx->cz - cx->oz)})) + 1.0;
    const double err = 2.0 * c * std::sqrt(3.0) * (2.0 * M * u + c * u) + 4.0 * c * c * u;
    p.guard = static_cast<float>(4.0 * err + 1e-6);
    // the spheres' margin: their FP32 images and transforms are off by a few M u
    p.reach = static_cast<float>(cutoff + 0.05 + 32.0 * M * u);
  }
  p.counts = d_counts;
  p.lists = d_lists;
  p.cap = cap;
  p.ubits = d_ubits;
  p.rows = d_rows;
  p.row_words = row_words;
  p.err = ctx->d_err;
  // whole blocks of ligand residues per unit, halves where the blocks give
  // every resident warp less than six and quarters where less than one (whole
  // calls at units of 2 / 4 / 8 residues: 183 poses of 130 x 90 residues 139 /
  // 144 / 165 us, 1,500 poses 443 / 426 / 442; 800 poses of 1,000 x 300 residues
  // 557 / 519 / 500); CTAs per pose so that few poses of many residues fill the
  // SMs, too
  const long long warps = 6LL * kContactWarps * ctx->sm_count, blocks = (t->GL + kLigBlock - 1) / kLigBlock;
  p.unit = n * blocks >= 6 * warps ? kLigBlock : (n * blocks >= warps ? kLigBlock / 2 : kLigBlock / 4);
  const long long units = (t->GL + p.unit - 1) / p.unit;
  p.parts = static_cast<int>(std::max(1LL, std::min((units + kContactWarps - 1) / kContactWarps,
                                                    6LL * ctx->sm_count / n)));
  k_contacts<<<static_cast<unsigned>(n) * p.parts, kContactWarps * 32, 0, st>>>(p);
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(ctx, e, "contacts launch");
  return GD_OK;
}

// Contacts of n poses through k_contacts: (receptor residue group * GL +
// ligand residue group) entries, flat with per-pose offsets loffs (n + 1
// entries).
static gd_status contacts_fast(gd_complex *cx, ClusterTopo *t, const std::vector<gd_pose_frame> &frames, int n,
                               double cutoff, double maxd, std::vector<uint32_t> &flat,
                               std::vector<long long> &loffs) {
  gd_context *ctx = cx->ctx;
  cudaStream_t st = ctx->stream;
  const size_t fb = al256(sizeof(gd_pose_frame) * n), cb = al256(sizeof(int) * n), ob = al256(sizeof(long long) * (n + 1));
  std::vector<int> counts(n);
  for (int cap = list_cap(ctx, t, n);;) {
    const size_t lb = al256(sizeof(uint32_t) * static_cast<size_t>(n) * cap);
    gd_status s = ensure_scratch(ctx, fb + cb + ob + lb, 0);
    if (s == GD_ERR_OOM && n > 64) {  // half of the poses at a time
      std::vector<gd_pose_frame> part(frames.begin(), frames.begin() + n / 2);
      s = contacts_fast(cx, t, part, n / 2, cutoff, maxd, flat, loffs);
      if (s != GD_OK) return s;
      std::vector<uint32_t> more;
      std::vector<long long> offs;
      part.assign(frames.begin() + n / 2, frames.begin() + n);
      s = contacts_fast(cx, t, part, n - n / 2, cutoff, maxd, more, offs);
      if (s != GD_OK) return s;
      const long long at = loffs.back();
      flat.insert(flat.end(), more.begin(), more.end());
      for (size_t i = 1; i < offs.size(); ++i) loffs.push_back(at + offs[i]);
      ctx->last_error.clear();  // the refused allocation is not this call's failure
      return GD_OK;
    }
    if (s != GD_OK) return s;
    char *base = static_cast<char *>(ctx->d_scratch);
    gd_pose_frame *d_frames = reinterpret_cast<gd_pose_frame *>(base);
    int *d_counts = reinterpret_cast<int *>(base + fb);
    long long *d_offs = reinterpret_cast<long long *>(base + fb + cb);
    uint32_t *d_lists = reinterpret_cast<uint32_t *>(base + fb + cb + ob);
    cudaError_t e = cudaMemcpyAsync(d_frames, frames.data(), sizeof(gd_pose_frame) * n, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "contacts setup");
    s = launch_contacts(cx, t, d_frames, n, cutoff, maxd, d_counts, d_lists, cap, nullptr, st);
    if (s != GD_OK) return s;
    e = cudaMemcpyAsync(counts.data(), d_counts, sizeof(int) * n, cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "contacts");
    if ((s = finish_stream(ctx, st, "contacts")) != GD_OK) return s;
    const int most = *std::max_element(counts.begin(), counts.end());
    if (most > cap) {  // once more with room for the largest pose
      cap = most;
      continue;
    }
    loffs.assign(n + 1, 0);
    for (int i = 0; i < n; ++i) loffs[i + 1] = loffs[i] + counts[i];
    flat.resize(static_cast<size_t>(loffs[n]));
    ctx->last_contacts = 2;
    if (loffs[n] == 0) return GD_OK;
    void *d_flat = nullptr;
    const size_t flat_b = sizeof(uint32_t) * flat.size();
    s = dev_alloc(ctx, flat_b, &d_flat);
    if (s == GD_ERR_OOM) {  // no room to gather them on the device: the lists up to the longest one
      std::vector<uint32_t> all(static_cast<size_t>(n) * most);
      e = cudaMemcpy2DAsync(all.data(), sizeof(uint32_t) * most, d_lists, sizeof(uint32_t) * cap, sizeof(uint32_t) * most, n,
                            cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) return cuda_fail(ctx, e, "contact lists");
      for (int i = 0; i < n; ++i)
        std::copy_n(all.begin() + static_cast<size_t>(i) * most, counts[i], flat.begin() + loffs[i]);
      ctx->last_error.clear();  // the refused allocation is not this call's failure
      return GD_OK;
    }
    if (s != GD_OK) return s;
    e = cudaMemcpyAsync(d_offs, loffs.data(), sizeof(long long) * (n + 1), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
      k_compact_lists<<<std::min(n, ctx->sm_count * 8), 128, 0, st>>>(d_lists, d_counts, d_offs, n, cap,
                                                                       static_cast<uint32_t *>(d_flat));
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(flat.data(), d_flat, flat_b, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    dev_free(ctx, d_flat, flat_b);
    return e == cudaSuccess ? GD_OK : cuda_fail(ctx, e, "contact list gather");
  }
}

// Orders the contacts of poses of two molecules of one chain each: keys by the
// residues of the smaller chain, then by the other's.  A pose's contacts are set
// as bits at their keys' ranks and read off in order; where the bits would be many
// more than the contacts, the keys are sorted.  The lists come in no order: with a
// sort for every pose 200 poses of 50 x 76 residues took 3.2 ms, with lists in the
// order of the residues and a sort of those 1.4, so 0.88.
class KeyOrder {
 public:
  explicit KeyOrder(const ClusterTopo *t) : t_(t), rec_first_((t->rg_key[0] >> 16) < (t->lg_key[0] >> 16)) {
    hi_.resize(rec_first_ ? t->GR : t->GL);
    lo_.resize(rec_first_ ? t->GL : t->GR);
    auto put = [](std::vector<int64_t> &v, const std::vector<int64_t> &key, const std::vector<int> &rank, int shift) {
      for (size_t g = 0; g < v.size(); ++g)
        v[rank[g]] = ((key[g] >> 16) << (16 + shift)) | ((key[g] & 0xffff) << shift);
    };
    put(hi_, rec_first_ ? t->rg_key : t->lg_key, rec_first_ ? t->rg_rank : t->lg_rank, 32);
    put(lo_, rec_first_ ? t->lg_key : t->rg_key, rec_first_ ? t->lg_rank : t->rg_rank, 0);
    row_ = (lo_.size() + 63) / 64;
  }
  void append(const uint32_t *v, size_t n, std::vector<uint64_t> &bits, std::vector<int64_t> &out) const {
    const uint32_t GL = static_cast<uint32_t>(t_->GL);
    const size_t words = hi_.size() * row_;
    const bool by_bits = words <= 16 * n;
    if (by_bits) bits.resize(words, 0);  // (all zero between poses)
    const size_t from = out.size();
    for (size_t k = 0; k < n; ++k) {
      const uint32_t rg = v[k] / GL, lg = v[k] % GL;
      const size_t a = rec_first_ ? t_->rg_rank[rg] : t_->lg_rank[lg], b = rec_first_ ? t_->lg_rank[lg] : t_->rg_rank[rg];
      if (by_bits) bits[a * row_ + (b >> 6)] |= uint64_t(1) << (b & 63);
      else out.push_back(hi_[a] | lo_[b]);
    }
    if (!by_bits) {
      std::sort(out.begin() + from, out.end());
      return;
    }
    out.resize(from + n);
    size_t at = from;
    for (size_t a = 0; a < hi_.size(); ++a)
      for (size_t w = 0; w < row_; ++w) {
        uint64_t &word = bits[a * row_ + w];
        for (uint64_t x = word; x; x &= x - 1) out[at++] = hi_[a] | lo_[w * 64 + __builtin_ctzll(x)];
        word = 0;
      }
  }

 private:
  const ClusterTopo *t_;
  bool rec_first_;
  std::vector<int64_t> hi_, lo_;  // a key's halves by rank
  size_t row_;                    // words a row of bits
};

// Contact keys of n poses (sorted per pose) into a host vector + offsets:
// through k_contacts when the topology allows it (and GD_TUNE_CONTACTS does not
// ask for the other), else through k_contacts_rl.  Both decide every atom pair
// exactly.
gd_status pose_contacts_host(gd_complex *cx, const double *genes, int n, double cutoff, std::vector<int64_t> &keys,
                             std::vector<int64_t> &offs) {
  gd_context *ctx = cx->ctx;
  PhaseTimer pt_all("contacts: total");
  ClusterTopo *t = nullptr;
  gd_status s = get_topo(cx, &t);
  if (s != GD_OK) return s;
  const Thresholds thr = make_thresholds(cutoff);
  if (t->multi_chain_rec && t->rr_cutoff != cutoff) {
    t->rr_keys.clear();
    intra_contacts(t->r_by_key.key, t->r_by_key.off, t->r_by_key.atoms, cx->h_rx.data(), cx->h_ry.data(), cx->h_rz.data(),
                   thr.contact_le, t->rr_keys);
    t->rr_cutoff = cutoff;
  }
  std::vector<gd_pose_frame> frames(n);
  gd_make_frames(genes, n, frames.data());
  const long long pairs = static_cast<long long>(t->GR) * t->GL;
  int cap = static_cast<int>(std::min<long long>(std::max<long long>(pairs, 1), 2048));
  std::vector<int> counts(n);
  std::vector<uint32_t> flat;
  std::vector<long long> loffs(n + 1, 0);
  const bool fast = ctx->tune_contacts != 1 && n > 0 && fast_contacts_ok(t);
  if (fast) {
    s = contacts_fast(cx, t, frames, n, cutoff, max_displacement(genes, n), flat, loffs);
    if (s != GD_OK) return s;
  } else {
    ctx->last_contacts = 1;
  }
  for (int attempt = 0; attempt < 2 && !fast; ++attempt) {
    const size_t fb = sizeof(gd_pose_frame) * n, cb = sizeof(int) * n,
                 lb = sizeof(uint32_t) * static_cast<size_t>(n) * cap, ob = sizeof(long long) * (n + 1);
    auto al = [](size_t b) { return (b + 255) / 256 * 256; };
    s = ensure_scratch(ctx, al(fb) + al(cb) + al(lb) + al(ob) + al(lb), 0);
    if (s != GD_OK) return s;
    char *base = static_cast<char *>(ctx->d_scratch);
    gd_pose_frame *d_frames = reinterpret_cast<gd_pose_frame *>(base);
    int *d_counts = reinterpret_cast<int *>(base + al(fb));
    uint32_t *d_lists = reinterpret_cast<uint32_t *>(base + al(fb) + al(cb));
    long long *d_offs = reinterpret_cast<long long *>(base + al(fb) + al(cb) + al(lb));
    uint32_t *d_flat = reinterpret_cast<uint32_t *>(base + al(fb) + al(cb) + al(lb) + al(ob));
    cudaError_t e = cudaMemcpyAsync(d_frames, frames.data(), fb, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_counts, 0, cb, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "contacts setup");
    if (pairs > 0) {
      ContactParams p{};
      p.rx = t->d_rx;
      p.ry = t->d_ry;
      p.rz = t->d_rz;
      p.rg_off = t->d_rg_off;
      p.rg_sph = t->d_rg_sph;
      p.rg_chain = t->d_rg_chain;
      p.lx = t->d_lx;
      p.ly = t->d_ly;
      p.lz = t->d_lz;
      p.lg_off = t->d_lg_off;
      p.lg_sph = t->d_lg_sph;
      p.lg_chain = t->d_lg_chain;
      p.GR = t->GR;
      p.GL = t->GL;
      p.cx = cx->cx;
      p.cy = cx->cy;
      p.cz = cx->cz;
      p.ox = cx->ox;
      p.oy = cx->oy;
      p.oz = cx->oz;
      p.frames = d_frames;
      p.n = n;
      p.t_le = thr.contact_le;
      p.reach = static_cast<float>(cutoff) + 0.05f;
      p.counts = d_counts;
      p.lists = d_lists;
      p.cap = cap;
      const long long items = static_cast<long long>(n) * t->GL;
      const int grid = static_cast<int>(std::min<long long>((items + kContactWarps - 1) / kContactWarps,
                                                            static_cast<long long>(ctx->sm_count) * 16));
      k_contacts_rl<<<grid, kContactWarps * 32, 0, ctx->stream>>>(p);
      if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(ctx, e, "contacts kernel launch");
    }
    e = cudaMemcpyAsync(counts.data(), d_counts, cb, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "contacts kernel");
    trace("contacts: kernel + counts", std::chrono::duration<double>(std::chrono::steady_clock::now() - pt_all.t0).count());
    const int maxc = n > 0 ? *std::max_element(counts.begin(), counts.end()) : 0;
    if (maxc > cap) {  // rerun once with room for the largest pose
      cap = maxc;
      continue;
    }
    for (int i = 0; i < n; ++i) loffs[i + 1] = loffs[i] + counts[i];
    flat.resize(static_cast<size_t>(loffs[n]));
    if (loffs[n] > 0) {
      e = cudaMemcpyAsync(d_offs, loffs.data(), ob, cudaMemcpyHostToDevice, ctx->stream);
      if (e != cudaSuccess) return cuda_fail(ctx, e, "H2D offsets");
      k_compact_lists<<<std::min(n, ctx->sm_count * 8), 128, 0, ctx->stream>>>(d_lists, d_counts, d_offs, n, cap,
                                                                                 d_flat);
      e = cudaMemcpyAsync(flat.data(), d_flat, sizeof(uint32_t) * flat.size(), cudaMemcpyDeviceToHost, ctx->stream);
      if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
      if (e != cudaSuccess) return cuda_fail(ctx, e, "contact list gather");
    }
    break;
  }
  PhaseTimer pt_keys("contacts: host keys");
  // each pose's keys on up to 16 threads (contiguous pose ranges), then
  // concatenated in pose order
  const int nth = n >= 256 ? static_cast<int>(std::max(1u, std::min(16u, std::thread::hardware_concurrency()))) : 1;
  std::vector<std::vector<int64_t>> part(nth);
  std::vector<int64_t> cnt(n, 0);
  if (fast && pairs > 0) {
    const KeyOrder order(t);
    auto work = [&](int q) {
      const int i0 = static_cast<int>(static_cast<long long>(n) * q / nth),
                i1 = static_cast<int>(static_cast<long long>(n) * (q + 1) / nth);
      std::vector<uint64_t> bits;
      part[q].reserve(static_cast<size_t>(loffs[i1] - loffs[i0]));
      for (int i = i0; i < i1; ++i)
        order.append(flat.data() + loffs[i], static_cast<size_t>(loffs[i + 1] - loffs[i]), bits, part[q]);
    };
    if (nth == 1) {
      work(0);
      keys.swap(part[0]);
    } else {
      std::vector<std::thread> th;
      for (int q = 0; q < nth; ++q) th.emplace_back(work, q);
      for (auto &x : th) x.join();
      keys.clear();
      keys.reserve(static_cast<size_t>(loffs[n]));
      for (const auto &v : part) keys.insert(keys.end(), v.begin(), v.end());
    }
    offs.assign(loffs.begin(), loffs.end());
    return GD_OK;
  }
  auto work = [&](int q) {
    const int i0 = static_cast<int>(static_cast<long long>(n) * q / nth),
              i1 = static_cast<int>(static_cast<long long>(n) * (q + 1) / nth);
    std::vector<int64_t> pk;
    std::vector<double> tx, ty, tz;
    for (int i = i0; i < i1; ++i) {
      pk.clear();
      for (long long k = loffs[i]; k < loffs[i + 1]; ++k) {
        const uint32_t v = flat[k];
        pk.push_back(canon(t->rg_key[v / t->GL], t->lg_key[v % t->GL]));
      }
      pk.insert(pk.end(), t->rr_keys.begin(), t->rr_keys.end());
      if (t->multi_chain_lig) {
        tx.resize(cx->nl);
        ty.resize(cx->nl);
        tz.resize(cx->nl);
        for (int a : t->l_atoms)
          xform_host(frames[i], cx->cx, cx->cy, cx->cz, cx->h_lx[a], cx->h_ly[a], cx->h_lz[a], tx[a], ty[a], tz[a]);
        intra_contacts(t->l_by_key.key, t->l_by_key.off, t->l_by_key.atoms, tx.data(), ty.data(), tz.data(), thr.contact_le, pk);
      }
      std::sort(pk.begin(), pk.end());
      pk.erase(std::unique(pk.begin(), pk.end()), pk.end());
      part[q].insert(part[q].end(), pk.begin(), pk.end());
      cnt[i] = static_cast<int64_t>(pk.size());
    }
  };
  if (nth == 1) {
    work(0);
  } else {
    std::vector<std::thread> th;
    for (int q = 0; q < nth; ++q) th.emplace_back(work, q);
    for (auto &x : th) x.join();
  }
  offs.assign(n + 1, 0);
  for (int i = 0; i < n; ++i) offs[i + 1] = offs[i] + cnt[i];
  keys.clear();
  keys.reserve(static_cast<size_t>(offs[n]));
  for (const auto &v : part) keys.insert(keys.end(), v.begin(), v.end());
  return GD_OK;
}

gd_status cluster_sets(gd_context *ctx, const int64_t *keys, const int64_t *offs, int n, const gd_cluster_cfg &cfg,
                       int32_t *n_clusters, int32_t *centers, int32_t *sizes, int32_t *members) {
  *n_clusters = 0;
  if (n <= 0) return GD_OK;
  PhaseTimer pt_all("fcc: total");
  // compacted contact universe, each pose's contacts as universe indices
  // (distinct, ascending) and the number of poses per contact; the host work
  // runs on up to 16 threads (poses split in contiguous ranges)
  const size_t nk = static_cast<size_t>(offs[n]);
  const int nth = nk >= (1u << 16) ? static_cast<int>(std::max(1u, std::min(16u, std::thread::hardware_concurrency()))) : 1;
  auto parallel = [nth](int count, const std::function<void(int, int, int)> &f) {
    if (nth == 1) return f(0, 0, count);
    std::vector<std::thread> th;
    for (int t = 0; t < nth; ++t)
      th.emplace_back(f, t, static_cast<int>(static_cast<long long>(count) * t / nth),
                      static_cast<int>(static_cast<long long>(count) * (t + 1) / nth));
    for (auto &x : th) x.join();
  };
  std::vector<int64_t> uni(keys, keys + nk);
  {
    // sorted runs per thread, then pairwise merges
    std::vector<size_t> cut(nth + 1);
    for (int t = 0; t <= nth; ++t) cut[t] = nk * t / nth;
    parallel(nth, [&](int, int t0, int t1) {
      for (int t = t0; t < t1; ++t) std::sort(uni.begin() + cut[t], uni.begin() + cut[t + 1]);
    });
    for (int w = 1; w < nth; w *= 2)
      for (int t = 0; t + w < nth; t += 2 * w)
        std::inplace_merge(uni.begin() + cut[t], uni.begin() + cut[t + w], uni.begin() + cut[std::min(nth, t + 2 * w)]);
    uni.erase(std::unique(uni.begin(), uni.end()), uni.end());
  }
  const int U = static_cast<int>(uni.size());
  std::vector<int> ui(nk);
  std::vector<int64_t> uoff(n + 1, 0);
  std::vector<int> sz(n), kc(std::max(U, 1), 0);
  parallel(n, [&](int, int i0, int i1) {
    for (int i = i0; i < i1; ++i) {
      const size_t o = static_cast<size_t>(offs[i]);
      size_t m = o;
      for (int64_t k = offs[i]; k < offs[i + 1]; ++k)
        ui[m++] = static_cast<int>(std::lower_bound(uni.begin(), uni.end(), keys[k]) - uni.begin());
      if (!std::is_sorted(ui.begin() + o, ui.begin() + m)) std::sort(ui.begin() + o, ui.begin() + m);
      sz[i] = static_cast<int>(std::unique(ui.begin() + o, ui.begin() + m) - (ui.begin() + o));
    }
  });
  // each pose's distinct indices packed to the front of its range
  for (int i = 0; i < n; ++i) {
    const size_t o = static_cast<size_t>(offs[i]), d = static_cast<size_t>(uoff[i]);
    if (d != o) std::copy(ui.begin() + o, ui.begin() + o + sz[i], ui.begin() + d);
    for (int k = 0; k < sz[i]; ++k) ++kc[ui[d + k]];
    uoff[i + 1] = uoff[i] + sz[i];
  }
  const int W = std::max(1, (U + 63) / 64);
  const int aw = (n + 31) / 32;
  auto al = [](size_t b) { return (b + 255) / 256 * 256; };
  // pair counts: bitsets, or the poses of each contact (postings) when the
  // contacts are spread thin (GD_TUNE_FCC; the same cost model as the device
  // clustering path)
  double work = 0.0;
  for (int u = 0; u < U; ++u) work += 0.5 * static_cast<double>(kc[u]) * (kc[u] - 1);
  const double bits_work = 0.5 * static_cast<double>(n) * (n + 1) * W;
  bool postings = n <= 16384 && (ctx->tune_fcc == 2 || (ctx->tune_fcc == 0 && bits_work > 2e10 && 80.0 * work < bits_work));
  const size_t sb = sizeof(int) * n, ab = sizeof(uint32_t) * static_cast<size_t>(n) * aw, gb = greedy_bytes(n);
  cudaStream_t st = ctx->stream;
  gd_status s = GD_OK;
  if (postings) {
    const size_t memb = static_cast<size_t>(uoff[n]);
    std::vector<int> poff(U + 1, 0), list(std::max<size_t>(memb, 1));
    for (int u = 0; u < U; ++u) poff[u + 1] = poff[u] + kc[u];
    std::vector<int> cur(poff.begin(), poff.end() - 1);
    for (int i = 0; i < n; ++i)
      for (int64_t k = uoff[i]; k < uoff[i + 1]; ++k) list[cur[ui[k]]++] = i;
    const size_t ob = sizeof(int) * (U + 1), kb = sizeof(int) * std::max(U, 1), lb = sizeof(int) * list.size(),
                 cb = sizeof(uint32_t) * static_cast<size_t>(n) * n;
    const size_t total = al(ob) + al(kb) + al(lb) + al(cb) + al(sb) + al(ab) + gb;
    void *buf = nullptr;
    s = dev_alloc(ctx, total, &buf);
    if (s != GD_OK && ctx->tune_fcc != 2) {
      postings = false;  // no room for the n x n counts: the bitsets
      ctx->last_error.clear();
    } else if (s != GD_OK) {
      return s;
    }
    if (postings) {
      trace("fcc: universe + postings (host)",
            std::chrono::duration<double>(std::chrono::steady_clock::now() - pt_all.t0).count());
      const auto t_k = std::chrono::steady_clock::now();
      char *b = static_cast<char *>(buf);
      int *d_off = reinterpret_cast<int *>(b);
      int *d_kc = reinterpret_cast<int *>(b + al(ob));
      int *d_list = reinterpret_cast<int *>(b + al(ob) + al(kb));
      uint32_t *d_common = reinterpret_cast<uint32_t *>(b + al(ob) + al(kb) + al(lb));
      int *d_sz = reinterpret_cast<int *>(b + al(ob) + al(kb) + al(lb) + al(cb));
      uint32_t *d_adj = reinterpret_cast<uint32_t *>(b + al(ob) + al(kb) + al(lb) + al(cb) + al(sb));
      cudaError_t e = cudaMemcpyAsync(d_off, poff.data(), ob, cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) e = cudaMemcpyAsync(d_kc, kc.data(), kb, cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) e = cudaMemcpyAsync(d_list, list.data(), lb, cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) e = cudaMemcpyAsync(d_sz, sz.data(), sb, cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) e = cudaMemsetAsync(d_common, 0, cb, st);
      if (e == cudaSuccess) e = cudaMemsetAsync(d_adj, 0, ab, st);
      if (e == cudaSuccess && U > 0)
        k_post_pairs<<<std::max(1, std::min((U + 7) / 8, ctx->sm_count * 16)), 256, 0, st>>>(d_off, d_kc, d_list, U, n,
                                                                                            d_common);
      if (e == cudaSuccess) {
        k_post_decide<<<std::min(n, ctx->sm_count * 16), 256, 0, st>>>(d_common, d_sz, n, cfg.fcc_cutoff,
                                                                       cfg.fcc_cutoff * cfg.strictness, d_adj, aw, 0);
        e = cudaGetLastError();
      }
      s = e == cudaSuccess ? greedy_clusters(ctx, d_adj, n, aw, cfg.min_cluster_size, b + total - gb, n_clusters, centers,
                                             sizes, members)
                           : cuda_fail(ctx, e, "FCC postings");
      if (s != GD_OK) cudaStreamSynchronize(st);
      dev_free(ctx, buf, total);
      if (s == GD_OK) ctx->last_fcc = 2;
      trace("fcc: kernels + transfers", std::chrono::duration<double>(std::chrono::steady_clock::now() - t_k).count());
      return s;
    }
  }
  std::vector<unsigned long long> bits(static_cast<size_t>(n) * W, 0ull);
  parallel(n, [&](int, int i0, int i1) {
    for (int i = i0; i < i1; ++i)
      for (int64_t k = uoff[i]; k < uoff[i + 1]; ++k)
        bits[static_cast<size_t>(i) * W + ui[k] / 64] |= 1ull << (ui[k] % 64);
  });
  const size_t bb = sizeof(unsigned long long) * bits.size();
  s = ensure_scratch(ctx, al(bb) + al(sb) + al(ab) + 256 + gb, 0);
  if (s != GD_OK) return s;
  char *base = static_cast<char *>(ctx->d_scratch);
  unsigned long long *d_bits = reinterpret_cast<unsigned long long *>(base);
  int *d_sz = reinterpret_cast<int *>(base + al(bb));
  uint32_t *d_adj = reinterpret_cast<uint32_t *>(base + al(bb) + al(sb));
  int *d_info = reinterpret_cast<int *>(base + al(bb) + al(sb) + al(ab));
  trace("fcc: universe + bitsets (host)",
        std::chrono::duration<double>(std::chrono::steady_clock::now() - pt_all.t0).count());
  const auto t_k = std::chrono::steady_clock::now();
  cudaError_t e = cudaMemcpyAsync(d_bits, bits.data(), bb, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_sz, sz.data(), sb, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_info, &U, sizeof(int), cudaMemcpyHostToDevice, st);
  FccParams p{};
  p.bits = d_bits;
  p.sizes = d_sz;
  p.info = d_info;
  p.n = n;
  p.stride = W;
  p.c = cfg.fcc_cutoff;
  p.cs = cfg.fcc_cutoff * cfg.strictness;
  p.adj = d_adj;
  p.adj_words = aw;
  if (e == cudaSuccess) e = launch_fcc(p, st);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "FCC kernel launch");
  s = greedy_clusters(ctx, d_adj, n, aw, cfg.min_cluster_size, base + al(bb) + al(sb) + al(ab) + 256, n_clusters, centers,
                      sizes, members);
  if (s != GD_OK) return s;
  ctx->last_fcc = 1;
  trace("fcc: kernels + transfers", std::chrono::duration<double>(std::chrono::steady_clock::now() - t_k).count());
  return GD_OK;
}

// Clusters of n poses from a bit per residue pair and pose, without lists and
// the universe: for contexts whose budget has no room for those.  The pair
// counts run over every residue pair, so it is the slower form.
static gd_status cluster_bits(gd_complex *cx, ClusterTopo *t, const gd_pose_frame *frames, int n, double maxd,
                              const gd_cluster_cfg &cfg, int c0, int32_t *n_clusters, int32_t *centers, int32_t *sizes,
                              int32_t *members) {
  gd_context *ctx = cx->ctx;
  cudaStream_t st = ctx->stream;
  const long long pairs = static_cast<long long>(t->GR) * t->GL;
  if (pairs > INT32_MAX) return GD_ERR_OOM;
  const int wide = std::max(1, static_cast<int>((pairs + 63) / 64)), aw = (n + 31) / 32;
  const size_t fb = al256(sizeof(gd_pose_frame) * n), cb = al256(sizeof(int) * n),
               rb = al256(sizeof(unsigned long long) * static_cast<size_t>(wide) * n),
               adj_b = al256(sizeof(uint32_t) * static_cast<size_t>(n) * aw);
  gd_status s = ensure_scratch(ctx, fb + cb + 256 + rb + adj_b + greedy_bytes(n), 0);
  if (s != GD_OK) return s;
  char *b = static_cast<char *>(ctx->d_scratch);
  gd_pose_frame *d_frames = reinterpret_cast<gd_pose_frame *>(b);
  FccParams fp{};
  int *d_counts = reinterpret_cast<int *>(b + fb), *d_info = reinterpret_cast<int *>(b + fb + cb);
  fp.sizes = d_counts;
  fp.info = d_info;
  fp.bits = reinterpret_cast<unsigned long long *>(b + fb + cb + 256);
  fp.adj = reinterpret_cast<uint32_t *>(b + fb + cb + 256 + rb);
  fp.n = n;
  fp.stride = wide;
  fp.c = cfg.fcc_cutoff;
  fp.cs = cfg.fcc_cutoff * cfg.strictness;
  fp.adj_words = aw;
  fp.c0 = c0;
  ctx->h_info[0] = static_cast<int>(pairs);
  cudaError_t e = cudaMemcpyAsync(d_frames, frames, sizeof(gd_pose_frame) * n, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_info, ctx->h_info, sizeof(int), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(b + fb + cb + 256, 0, rb, st);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "contacts setup");
  s = launch_contacts(cx, t, d_frames, n, cfg.contact_distance, maxd, d_counts, nullptr, 0, nullptr, st,
                      reinterpret_cast<uint32_t *>(b + fb + cb + 256), 2LL * wide);
  if (s != GD_OK) return s;
  if ((e = launch_fcc(fp, st)) != cudaSuccess) return cuda_fail(ctx, e, "FCC on the device");
  s = greedy_clusters(ctx, fp.adj, n, aw, cfg.min_cluster_size, b + fb + cb + 256 + rb + adj_b, n_clusters, centers, sizes, members);
  if (s != GD_OK) return s;
  ctx->last_contacts = 2;
  ctx->last_fcc = 1;
  ctx->last_error.clear();  // the refused allocation is not this call's failure
  return GD_OK;
}

// cluster_structures on the device for receptors and ligands that share no
// residue: contact lists, their union, FCC over bitsets or postings, greedy
// clustering.  Returns GD_ERR_STATE when the topology calls for the general
// path.
gd_status cluster_device(gd_complex *cx, const double *genes, int n, const gd_cluster_cfg &cfg, int32_t *n_clusters,
                         int32_t *centers, int32_t *sizes, int32_t *members) {
  gd_context *ctx = cx->ctx;
  PhaseTimer pt_all("cluster (device): total");
  ClusterTopo *t = nullptr;
  gd_status s = get_topo(cx, &t);
  if (s != GD_OK) return s;
  if (!fast_contacts_ok(t, true)) return GD_ERR_STATE;
  // contacts within one molecule across its chains are the same in every
  // pose (the receptor does not move; the ligand moves rigidly and its
  // decisions are checked to be far from the cutoff): a constant c0 in every
  // set size and pair count, outside the lists
  const Thresholds thr = make_thresholds(cfg.contact_distance);
  long long c0 = 0;
  if (t->multi_chain_rec) {
    if (t->rr_cutoff != cfg.contact_distance) {
      t->rr_keys.clear();
      intra_contacts(t->r_by_key.key, t->r_by_key.off, t->r_by_key.atoms, cx->h_rx.data(), cx->h_ry.data(), cx->h_rz.data(),
                     thr.contact_le, t->rr_keys);
      t->rr_cutoff = cfg.contact_distance;
    }
    c0 += static_cast<long long>(t->rr_keys.size());
  }
  if (t->multi_chain_lig) {
    if (t->ll_cutoff != cfg.contact_distance) {
      std::vector<int64_t> ll;
      bool unstable = false;
      intra_contacts(t->l_by_key.key, t->l_by_key.off, t->l_by_key.atoms, cx->h_lx.data(), cx->h_ly.data(), cx->h_lz.data(),
                     thr.contact_le, ll, &unstable);
      t->ll_count = static_cast<long long>(ll.size());
      t->ll_unstable = unstable;
      t->ll_cutoff = cfg.contact_distance;
    }
    if (t->ll_unstable) return GD_ERR_STATE;
    c0 += t->ll_count;
  }
  if (c0 > (1 << 30)) return GD_ERR_STATE;
  const long long words = pair_words(t), pairs = static_cast<long long>(t->GR) * t->GL;
  const int aw = (n + 31) / 32;
  const size_t fb = al256(sizeof(gd_pose_frame) * n), cb = al256(sizeof(int) * n), ub = al256(sizeof(uint32_t) * words),
               bb = al256(sizeof(int) * words), adj_b = al256(sizeof(uint32_t) * static_cast<size_t>(n) * aw);
  // small calls (rows over every residue pair, and the adjacency, within 16
  // MiB) take the bitsets without asking for the universe's size first
  const int wide = static_cast<int>(std::min<long long>((pairs + 63) / 64, INT32_MAX));
  const bool direct = ctx->tune_fcc != 2 &&
                      static_cast<size_t>(std::max(wide, 1)) * 8 * n + adj_b <= (size_t(16) << 20) &&
                      0.5 * static_cast<double>(n) * (n + 1) * wide <= 2e10;
  const size_t direct_b = direct ? al256(sizeof(unsigned long long) * static_cast<size_t>(std::max(wide, 1)) * n) + adj_b +
                                       greedy_bytes(n)
                                 : 0;
  cudaStream_t st = ctx->stream;
  int cap = list_cap(ctx, t, n), info[2] = {0, 0};
  gd_pose_frame *d_frames;
  int *d_counts, *d_base, *d_info;
  uint32_t *d_u, *d_lists;
  char *d_direct;
  auto t_step = std::chrono::steady_clock::now();
  // the frames are staged behind the place of the greedy pass's results
  const size_t res_b = n > kGreedyMax ? 0 : al256(greedy_bytes(n));
  const bool staged = fb <= kStageMax;
  if ((s = ensure_scratch(ctx, 0, staged ? res_b + fb : 0)) != GD_OK) return s;
  std::vector<gd_pose_frame> pageable(staged ? 0 : n);
  gd_pose_frame *frames =
      staged ? reinterpret_cast<gd_pose_frame *>(static_cast<char *>(ctx->h_pinned) + res_b) : pageable.data();
  double maxd = 0.0;
  frames_and_max_disp(genes, n, frames, &maxd);
  for (;;) {
    const size_t lb = al256(sizeof(uint32_t) * static_cast<size_t>(n) * cap);
    s = ensure_scratch(ctx, fb + cb + ub + bb + 256 + lb + direct_b, 0);
    if (s == GD_ERR_OOM)
      return cluster_bits(cx, t, frames, n, maxd, cfg, static_cast<int>(c0), n_clusters, centers, sizes, members);
    if (s != GD_OK) return s;
    char *b = static_cast<char *>(ctx->d_scratch);
    d_frames = reinterpret_cast<gd_pose_frame *>(b);
    d_counts = reinterpret_cast<int *>(b + fb);
    d_u = reinterpret_cast<uint32_t *>(b + fb + cb);
    d_base = reinterpret_cast<int *>(b + fb + cb + ub);
    d_info = reinterpret_cast<int *>(b + fb + cb + ub + bb);
    d_lists = reinterpret_cast<uint32_t *>(b + fb + cb + ub + bb + 256);
    d_direct = b + fb + cb + ub + bb + 256 + lb;
    cudaError_t e = cudaSuccess;
    if (n <= kDirectPoses && staged) d_frames = frames;  // read in place
    else e = cudaMemcpyAsync(d_frames, frames, sizeof(gd_pose_frame) * n, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "contacts setup");
    trace_step("cluster (device):   scratch + frames", st, t_step);
    s = launch_contacts(cx, t, d_frames, n, cfg.contact_distance, maxd, d_counts, d_lists, cap, d_u, st);
    if (s != GD_OK) return s;
    ctx->last_contacts = 2;
    trace_step("cluster (device):   k_contacts", st, t_step);
    k_scan<true><<<1, 1024, 0, st>>>(d_u, words, d_base, d_info, d_counts, n, d_info + 1, ctx->h_info);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(ctx, e, "contact union");
    trace_step("cluster (device):   union scan", st, t_step);
    FccParams fp{};
    fp.sizes = d_counts;
    fp.info = d_info;
    fp.n = n;
    fp.c = cfg.fcc_cutoff;
    fp.cs = cfg.fcc_cutoff * cfg.strictness;
    fp.adj_words = aw;
    fp.c0 = static_cast<int>(c0);
    auto rows = [&](unsigned long long *d_rows, int stride) -> cudaError_t {
      const int in_smem = stride <= kRowSmem;
      cudaError_t x = cudaSuccess;
      if (!in_smem) x = cudaMemsetAsync(d_rows, 0, sizeof(unsigned long long) * static_cast<size_t>(stride) * n, st);
      if (x != cudaSuccess) return x;
      k_rows<<<n, 256, in_smem ? sizeof(unsigned long long) * stride : 0, st>>>(d_lists, d_counts, cap, d_u, d_base, d_info,
                                                                              stride, in_smem, d_rows);
      return cudaGetLastError();
    };
    if (direct) {
      fp.stride = std::max(wide, 1);
      fp.bits = reinterpret_cast<unsigned long long *>(d_direct);
      char *d_adj = d_direct + al256(sizeof(unsigned long long) * static_cast<size_t>(fp.stride) * n);
      fp.adj = reinterpret_cast<uint32_t *>(d_adj);
      e = rows(reinterpret_cast<unsigned long long *>(d_direct), fp.stride);
      if (e == cudaSuccess) e = launch_fcc(fp, st);
      if (e != cudaSuccess) return cuda_fail(ctx, e, "FCC on the device");
      s = greedy_clusters(ctx, fp.adj, n, aw, cfg.min_cluster_size, d_adj + adj_b, n_clusters, centers, sizes, members);
      if (s != GD_OK) return s;
      if (ctx->h_info[1] <= cap) {
        ctx->last_fcc = 1;
        trace_step("cluster (device):   rows + fcc + greedy", st, t_step);
        return GD_OK;
      }
    } else {
      if ((s = finish_stream(ctx, st, "contact union")) != GD_OK) return s;
    }
    info[0] = ctx->h_info[0];
    info[1] = ctx->h_info[1];
    if (info[1] > cap) {  // once more with room for the pose with the most contacts
      cap = info[1];
      continue;
    }
    // pair counts: contact postings or bitsets (GD_TUNE_FCC; automatic: the
    // estimated cheaper one, postings only up to 16,384 poses, and considered
    // only when the bitsets would take more than ~2e10 word pairs, some 5 ms:
    // counting the postings costs a pass and a synchronisation)
    const int U = info[0], W = std::max(1, (U + 63) / 64);
    bool postings = ctx->tune_fcc == 2 && n <= 16384;
    const double bits_work = 0.5 * static_cast<double>(n) * (n + 1) * W;
    void *pre = nullptr;  // posting counts: kc[U], the work sum
    const size_t kc_b = al256(sizeof(int) * static_cast<size_t>(std::max(U, 1))), pre_b = kc_b + 256;
    if (ctx->tune_fcc != 1 && n <= 16384 && (ctx->tune_fcc == 2 || bits_work > 2e10)) {
      s = dev_alloc(ctx, pre_b, &pre);
      if (s != GD_OK && (s != GD_ERR_OOM || ctx->tune_fcc == 2)) return s;
    }
    if (s != GD_OK) {  // no room to count the postings: the bitsets
      ctx->last_error.clear();
      s = GD_OK;
    } else if (pre) {
      int *d_kc = static_cast<int *>(pre);
      unsigned long long *d_work = reinterpret_cast<unsigned long long *>(static_cast<char *>(pre) + kc_b), work = 0;
      e = cudaMemsetAsync(pre, 0, pre_b, st);
      if (e == cudaSuccess) {
        k_post_count<<<std::min(n, ctx->sm_count * 16), 256, 0, st>>>(d_lists, d_counts, cap, d_u, d_base, n, d_kc);
        k_post_work<<<std::max(1, std::min((U + 255) / 256, ctx->sm_count * 8)), 256, 0, st>>>(d_kc, U, d_work);
        e = cudaMemcpyAsync(&work, d_work, 8, cudaMemcpyDeviceToHost, st);
      }
      if (e == cudaSuccess) e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) {
        dev_free(ctx, pre, pre_b);
        return cuda_fail(ctx, e, "FCC posting counts");
      }
      // an atomic increment costs about as much as 80 word pairs of popcount
      if (ctx->tune_fcc == 0) postings = 80.0 * static_cast<double>(work) < bits_work;
    }
    if (!postings && pre) {
      dev_free(ctx, pre, pre_b);
      pre = nullptr;
    }
    // postings: offsets and cursors per contact, the lists (one entry per
    // (pose, contact)), the n x n common counts; bitsets: the rows
    size_t memberships = 0;
    if (postings) {
      std::vector<int> hsz(n);
      e = cudaMemcpy(hsz.data(), d_counts, sizeof(int) * n, cudaMemcpyDeviceToHost);
      if (e != cudaSuccess) {
        dev_free(ctx, pre, pre_b);
        return cuda_fail(ctx, e, "FCC posting sizes");
      }
      for (int v : hsz) memberships += static_cast<size_t>(v);
    }
    const size_t rows_b = al256(sizeof(unsigned long long) * static_cast<size_t>(W) * n);
    const size_t off_b = al256(sizeof(int) * (static_cast<size_t>(U) + 1)),
                 list_b = al256(sizeof(int) * std::max<size_t>(memberships, 1)),
                 common_b = al256(sizeof(uint32_t) * static_cast<size_t>(n) * n);
    size_t extra_b = (postings ? off_b + kc_b + list_b + common_b : rows_b) + adj_b + greedy_bytes(n);
    // up to 64 MiB from scratch that the context keeps for this (not where a
    // budget bounds what it may hold), else for this call alone
    const bool kept = !postings && ctx->budget == 0 && extra_b <= (size_t(64) << 20);
    void *extra = nullptr;
    if (kept) {
      s = ensure_cluster_scratch(ctx, extra_b);
      extra = ctx->d_cluster;
    } else {
      s = dev_alloc(ctx, extra_b, &extra);
    }
    if (s != GD_OK && postings && ctx->tune_fcc != 2) {
      // no room for the n x n counts: the bitsets after all
      dev_free(ctx, pre, pre_b);
      pre = nullptr;
      postings = false;
      extra_b = rows_b + adj_b + greedy_bytes(n);
      s = dev_alloc(ctx, extra_b, &extra);
      if (s == GD_OK) ctx->last_error.clear();  // the refused allocation is not this call's failure
    }
    if (s != GD_OK) {
      if (pre) dev_free(ctx, pre, pre_b);
      if (s == GD_ERR_OOM && !postings)
        return cluster_bits(cx, t, frames, n, maxd, cfg, static_cast<int>(c0), n_clusters, centers, sizes, members);
      return s;
    }
    ctx->last_fcc = postings ? 2 : 1;
    char *xp = static_cast<char *>(extra), *d_greedy = xp + extra_b - greedy_bytes(n);
    uint32_t *d_adj = reinterpret_cast<uint32_t *>(d_greedy - adj_b);
    if (postings) {
      int *d_kc = static_cast<int *>(pre);
      int *d_offs = reinterpret_cast<int *>(xp);
      int *d_cur = reinterpret_cast<int *>(xp + off_b);
      int *d_list = reinterpret_cast<int *>(xp + off_b + kc_b);
      uint32_t *d_common = reinterpret_cast<uint32_t *>(xp + off_b + kc_b + list_b);
      e = cudaMemsetAsync(d_cur, 0, kc_b, st);
      if (e == cudaSuccess) e = cudaMemsetAsync(d_common, 0, common_b + adj_b, st);
      if (e == cudaSuccess) {
        k_scan<false><<<1, 1024, 0, st>>>(reinterpret_cast<const uint32_t *>(d_kc), U, d_offs, d_offs + U, nullptr, 0, nullptr, nullptr);
        k_post_fill<<<std::min(n, ctx->sm_count * 16), 256, 0, st>>>(d_lists, d_counts, cap, d_u, d_base, n, d_offs, d_cur,
                                                                     d_list);
        k_post_pairs<<<std::max(1, std::min((U + 7) / 8, ctx->sm_count * 16)), 256, 0, st>>>(d_offs, d_kc, d_list, U, n,
                                                                                            d_common);
        k_post_decide<<<std::min(n, ctx->sm_count * 16), 256, 0, st>>>(d_common, d_counts, n, fp.c, fp.cs, d_adj, aw, fp.c0);
        e = cudaGetLastError();
      }
    } else {
      fp.bits = reinterpret_cast<unsigned long long *>(xp);
      fp.stride = W;
      fp.adj = d_adj;
      e = rows(reinterpret_cast<unsigned long long *>(xp), W);
      if (e == cudaSuccess) e = launch_fcc(fp, st);
    }
    s = e == cudaSuccess ? GD_OK : cuda_fail(ctx, e, "FCC on the device");
    trace_step(postings ? "cluster (device):   postings + fcc" : "cluster (device):   rows + fcc", st, t_step);
    if (s == GD_OK)
      s = greedy_clusters(ctx, d_adj, n, aw, cfg.min_cluster_size, d_greedy, n_clusters, centers, sizes, members);
    if (s != GD_OK) cudaStreamSynchronize(st);
    trace_step("cluster (device):   greedy", st, t_step);
    if (!kept) dev_free(ctx, extra, extra_b);
    if (pre) dev_free(ctx, pre, pre_b);
    return s;
  }
}

}  // namespace gd

using namespace gd;

static gd_cluster_cfg default_cfg() { return gd_cluster_cfg{5.0, 0.60, 0.75, 4}; }

extern "C" {

gd_status gd_pose_contacts(gd_complex *cx, const double *genes, int32_t n, int64_t *keys, int64_t cap,
                           int64_t *offsets) {
  gd::NvtxRange nvtx_range("gd_pose_contacts");
  if (!cx) return GD_ERR_INVALID_ARG;
  gd_context *ctx = cx->ctx;
  if (n < 0 || (n > 0 && (!genes || !offsets)) || cap < 0 || (cap > 0 && !keys))
    return fail(ctx, GD_ERR_INVALID_ARG, "bad genes/keys/offsets");
  cudaSetDevice(ctx->device);
  const ScratchUse use(ctx);
  std::vector<int64_t> k, o;
  gd_status s = pose_contacts_host(cx, genes, n, 5.0, k, o);
  if (s != GD_OK) return s;
  std::memcpy(offsets, o.data(), sizeof(int64_t) * (n + 1));
  if (static_cast<int64_t>(k.size()) > cap) return fail(ctx, GD_ERR_CAPACITY, "contact key buffer too small");
  if (!k.empty()) std::memcpy(keys, k.data(), sizeof(int64_t) * k.size());
  return GD_OK;
}

gd_status gd_cluster(gd_complex *cx, const double *genes, int32_t n, const gd_cluster_cfg *cfg, int32_t *n_clusters,
                     int32_t *centers, int32_t *sizes, int32_t *members) {
  gd::NvtxRange nvtx_range("gd_cluster");
  if (!cx) return GD_ERR_INVALID_ARG;
  gd_context *ctx = cx->ctx;
  if (n < 0 || (n > 0 && (!genes || !centers || !sizes || !members)) || !n_clusters)
    return fail(ctx, GD_ERR_INVALID_ARG, "bad cluster arguments");
  const gd_cluster_cfg c = cfg ? *cfg : default_cfg();
  *n_clusters = 0;
  if (n == 0) return GD_OK;  // cluster_structures on no structures
  cudaSetDevice(ctx->device);
  const ScratchUse use(ctx);
  gd_status s = cluster_device(cx, genes, n, c, n_clusters, centers, sizes, members);
  if (s != GD_ERR_STATE) return s;
  // multi-chain molecules or shared residues: contact keys on the host path
  std::vector<int64_t> k, o;
  s = pose_contacts_host(cx, genes, n, c.contact_distance, k, o);
  if (s != GD_OK) return s;
  return cluster_sets(ctx, k.data(), o.data(), n, c, n_clusters, centers, sizes, members);
}

gd_status gd_cluster_sets(gd_context *ctx, const int64_t *keys, const int64_t *offsets, int32_t n,
                          const gd_cluster_cfg *cfg, int32_t *n_clusters, int32_t *centers, int32_t *sizes,
                          int32_t *members) {
  gd::NvtxRange nvtx_range("gd_cluster_sets");
  if (!ctx) return GD_ERR_INVALID_ARG;
  if (n < 0 || (n > 0 && (!offsets || !centers || !sizes || !members)) || !n_clusters)
    return fail(ctx, GD_ERR_INVALID_ARG, "bad cluster arguments");
  if (n > 0 && offsets[n] > 0 && !keys) return fail(ctx, GD_ERR_INVALID_ARG, "null keys");
  cudaSetDevice(ctx->device);
  const gd_cluster_cfg c = cfg ? *cfg : default_cfg();
  const ScratchUse use(ctx);
  return cluster_sets(ctx, keys, offsets, n, c, n_clusters, centers, sizes, members);
}

}  // extern "C"
