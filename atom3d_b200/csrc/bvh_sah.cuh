// SAH refinement of the binary radix tree, one thread block per cluster.
//
// The Morton radix tree splits space at the midpoint planes of the centroid
// cube, which gives loose boxes near the leaves.  Every subtree of the radix
// tree with at most kSahMax triangles whose parent holds more (a "cluster")
// is rebuilt top-down with a binned surface-area heuristic (16 bins per
// axis, centroid binning, cost = A_left N_left + A_right N_right, ties to
// the lower axis and bin), down to single triangles:
//   * nodes of more than warp_max triangles are split by one block per
//     cluster (sah_cluster_kernel: shared-memory bins, block scans for a
//     stable partition);
//   * smaller nodes go on a list that all warps of the chip share
//     (sah_small_kernel); a warp splits them with bins of its own down to 32
//     triangles and builds the rest of the subtree, all its nodes of a level
//     at once, with one triangle a lane.
// The triangles' centroids and boxes are read from global memory (L2
// resident); the cluster's slice of the sorted face order is partitioned in
// place.  Partitions are stable, reductions are min/max/integer sums, so the
// result is deterministic.  A node with no valid split (coincident centroids) or
// deeper than kSahMaxDepth inside its cluster is split at its median position.
//
// Node numbering stays within the cluster's own index set.  A radix-tree
// subtree over sorted positions [f, l] uses the internal indices [f, l]
// except the end that is not its root; here the node whose split falls
// between local positions m-1 and m gets index f + m - 1 (+1 when the old
// root sat at l), which enumerates exactly that set, and the new root takes
// the old root's index (swapping with the node that would have had it), so
// the cluster's parent needs no update.  Leaves stay N + position; the
// cluster's slice of the sorted face order is rewritten.  Boxes are computed
// afterwards by the ordinary refit.
#pragma once

#include "a3d_common.cuh"

namespace a3d {
namespace {

constexpr int kSahMax = 16384;
constexpr int kSahBins = 16;
// largest node handed to a warp (warp_max): 256, from kSahWideFrom triangles in
// all on 512.  A block splits a cluster's larger nodes one after the other,
// about 12 us each whatever their size, while a warp's chain of 512 triangles
// takes longer than the rest of a small build (whole builds, at 128 / 256 /
// 512 / 1024: 20,480 triangles 861 / 869 / 1004 / 1394 us, 327,680: 1.57 /
// 1.47 / 1.53 / 1.87 ms, 1,310,720: 4.77 / 4.05 / 3.80 / 3.83 ms)
constexpr int kSahWarpMin = 256, kSahWarpWide = 512;
constexpr int64_t kSahWideFrom = 1 << 19;
// block size of the cluster kernel: 1024 threads when the clusters are
// about as many as the SMs (one mesh up to kSahMax x SMs triangles: each
// block's 32 warps share out its small nodes), 256 when there are many
// (batches: more blocks per SM, cheaper block-wide steps)
constexpr int kSahThreadsWide = 1024;
constexpr int kSahThreadsNarrow = 256;
constexpr int kSahMaxDepth = 48;
// nodes this small split at their median position: 2 = SAH all the way down
// (median splits at 8 and below cut a third of the 256-thread build time of
// the 1.31M-triangle tree but cost 21 more triangle tests per query, +1.2%
// query time)
constexpr int kSahTiny = 2;
constexpr int kSahCand = 3 * (kSahBins - 1);            // 45 split candidates
constexpr int kBinWords = 3 * kSahBins * 7;              // count, lo xyz, hi xyz
// a warp's pending nodes: one per level, at most kSahMaxDepth levels and the
// median splits of what is left below them
constexpr int kSahWarpStack = kSahMaxDepth + 16;
static_assert(kSahWarpWide <= (1 << 15), "median splits end within the stack");
constexpr int kSahBlockStack = kSahMax / (kSahWarpMin + 1) + 2;  // disjoint ranges above warp_max

// a node to split: local range [b, e) of its cluster, parent index (-1 for
// the cluster root), side in the parent, depth inside the cluster
struct SahNode {
  int b, e, parent, sd;  // sd = side | depth << 1
};

// a node of at most warp_max triangles waiting for a warp
struct SahSmall {
  SahNode node;
  int cluster;
};

template <int kThreads>
struct SahSmem {
  static constexpr int kWarps = kThreads / 32;
  uint32_t bins[kBinWords];
  SahNode bstack[kSahBlockStack];
  float red[kWarps][6];
  uint32_t wsum[kWarps];
  float cb[6];
  int nb, m, axis, kk, root_nat;
};

struct SahTree {
  int32_t* left;
  int32_t* right;
  int32_t* parent;
  int32_t* first;
  int32_t* last;
  int64_t n;  // total triangles (leaf j is n + j)
};

__device__ __forceinline__ float sah_half_area(float x0, float y0, float z0, float x1, float y1, float z1) {
  const float dx = x1 - x0, dy = y1 - y0, dz = z1 - z0;
  return dx * dy + dy * dz + dz * dx;
}

__device__ __forceinline__ int sah_bin(float c, float lo, float scale) {
  const int k = (int)((c - lo) * scale);
  return k < kSahBins - 1 ? k : kSahBins - 1;
}

// candidate `cand` (axis cand / 15, split after bin cand % 15) of the bins:
// cost and left count; cost = +inf when a side is empty or the axis is flat
__device__ __forceinline__ void sah_candidate(const uint32_t* bins, const float* cb, int cand, float& cost, int& nl) {
  cost = INFINITY;
  nl = 0;
  if (cand >= kSahCand) return;
  const int axis = cand / (kSahBins - 1), k = cand % (kSahBins - 1) + 1;
  if (!(cb[3 + axis] > cb[axis])) return;
  float l0 = INFINITY, l1 = INFINITY, l2 = INFINITY, u0 = -INFINITY, u1 = -INFINITY, u2 = -INFINITY;
  float r0 = INFINITY, r1 = INFINITY, r2 = INFINITY, v0 = -INFINITY, v1 = -INFINITY, v2 = -INFINITY;
  int cl = 0, cr = 0;
  for (int j = 0; j < kSahBins; ++j) {
    const uint32_t* w = bins + (axis * kSahBins + j) * 7;
    const int cnt = (int)w[0];
    if (cnt == 0) continue;
    const float a0 = float_unflip(w[1]), a1 = float_unflip(w[2]), a2 = float_unflip(w[3]);
    const float b0 = float_unflip(w[4]), b1 = float_unflip(w[5]), b2 = float_unflip(w[6]);
    if (j < k) {
      cl += cnt;
      l0 = fminf(l0, a0); l1 = fminf(l1, a1); l2 = fminf(l2, a2);
      u0 = fmaxf(u0, b0); u1 = fmaxf(u1, b1); u2 = fmaxf(u2, b2);
    } else {
      cr += cnt;
      r0 = fminf(r0, a0); r1 = fminf(r1, a1); r2 = fminf(r2, a2);
      v0 = fmaxf(v0, b0); v1 = fmaxf(v1, b1); v2 = fmaxf(v2, b2);
    }
  }
  if (cl == 0 || cr == 0) return;
  cost = sah_half_area(l0, l1, l2, u0, u1, u2) * (float)cl + sah_half_area(r0, r1, r2, v0, v1, v2) * (float)cr;
  nl = cl;
}

// the warp's best candidate (lowest cost, then lowest candidate index);
// returns the left count, 0 when no candidate is valid
__device__ __forceinline__ int sah_pick(const uint32_t* bins, const float* cb, int lane, int& axis, int& kk) {
  float cost0, cost1;
  int nl0, nl1;
  sah_candidate(bins, cb, lane, cost0, nl0);
  sah_candidate(bins, cb, lane + 32, cost1, nl1);
  float best = cost0;
  int bc = lane, bn = nl0;
  if (cost1 < best) { best = cost1; bc = lane + 32; bn = nl1; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float oc = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bc, o);
    const int on = __shfl_xor_sync(0xffffffffu, bn, o);
    if (oc < best || (oc == best && oi < bc)) { best = oc; bc = oi; bn = on; }
  }
  if (!(best < INFINITY)) return 0;
  axis = bc / (kSahBins - 1);
  kk = bc % (kSahBins - 1) + 1;
  return bn;
}

// the triangles' centroids and boxes, indexed by face id
struct SahPrims {
  const float4* __restrict__ cen;
  const float4* __restrict__ lo;
  const float4* __restrict__ hi;
};

__device__ __forceinline__ float sah_c(const float4& c, int a) { return a == 0 ? c.x : (a == 1 ? c.y : c.z); }

__device__ __forceinline__ void sah_bin_prim(uint32_t* bins, const SahPrims& P, uint32_t face, const float* cb,
                                             const float* scale) {
  const float4 c = __ldg(P.cen + face), lo = __ldg(P.lo + face), hi = __ldg(P.hi + face);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (!(cb[3 + a] > cb[a])) continue;
    uint32_t* w = bins + (a * kSahBins + sah_bin(sah_c(c, a), cb[a], scale[a])) * 7;
    atomicAdd(&w[0], 1u);
    atomicMin(&w[1], float_flip(lo.x));
    atomicMin(&w[2], float_flip(lo.y));
    atomicMin(&w[3], float_flip(lo.z));
    atomicMax(&w[4], float_flip(hi.x));
    atomicMax(&w[5], float_flip(hi.y));
    atomicMax(&w[6], float_flip(hi.z));
  }
}

__device__ __forceinline__ void sah_clear_bins(uint32_t* bins, int t, int nt) {
  for (int i = t; i < kBinWords; i += nt) {
    const int f = i % 7;
    bins[i] = f == 0 ? 0u : (f <= 3 ? 0xffffffffu : 0u);  // flipped +inf / -inf
  }
}

// index of the node of a cluster rooted at R over [f, l] that splits at local m
__device__ __forceinline__ int sah_label(int f, int m, int shift, int R, int root_nat, bool is_root) {
  const int nat = f + m - 1 + shift;
  if (is_root) return R;
  return nat == R ? root_nat : nat;
}

// writes the node's topology and the leaf children; returns the children
// that need processing through `push(b, e, side)`
template <typename Push>
__device__ __forceinline__ void sah_emit(const SahTree& T, int f, int b, int m, int e, int label, int plabel,
                                         int side, Push&& push) {
  T.first[label] = f + b;
  T.last[label] = f + e - 1;
  if (plabel >= 0) {
    T.parent[label] = plabel;
    if (side) T.right[plabel] = label;
    else T.left[plabel] = label;
  }
  if (m - b == 1) {
    const int leaf = (int)(T.n + f + b);
    T.left[label] = leaf;
    T.parent[leaf] = label;
  } else {
    push(b, m, 0);
  }
  if (e - m == 1) {
    const int leaf = (int)(T.n + f + m);
    T.right[label] = leaf;
    T.parent[leaf] = label;
  } else {
    push(m, e, 1);
  }
}

// One block per cluster (grid-stride over the device-side cluster list): the
// nodes above warp_max.  The cluster's slice of the sorted face order is
// partitioned in place (tmp: a scratch slice of the same positions); smaller
// nodes are appended to `small` (a cluster of n triangles has fewer than n of
// them), and root_nat[cluster] keeps the position its root would have had.
template <int kThreads>
__global__ void __launch_bounds__(kThreads)
    sah_cluster_kernel(const int32_t* __restrict__ clusters, const uint32_t* __restrict__ ncl, SahTree T,
                       uint32_t* __restrict__ order, uint32_t* __restrict__ tmp_all, SahSmall* __restrict__ small,
                       uint32_t* __restrict__ nsmall, int32_t* __restrict__ root_nat, int warp_max, SahPrims P) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char sah_raw[];
  constexpr int kWarps = kThreads / 32;
  SahSmem<kThreads>& S = *reinterpret_cast<SahSmem<kThreads>*>(sah_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned FULL = 0xffffffffu;
  const uint32_t count = *ncl;
  for (uint32_t ci = blockIdx.x; ci < count; ci += gridDim.x) {
    const int R = clusters[ci];
    const int f = T.first[R], l = T.last[R];
    const int n = l - f + 1;
    const int shift = (R == l) ? 1 : 0;
    uint32_t* ord = order + f;
    uint32_t* tmp = tmp_all + f;
    if (tid == 0) {
      S.nb = 0;
      const SahNode root{0, n, -1, 0};
      if (n > warp_max) S.bstack[S.nb++] = root;
      else small[atomicAdd(nsmall, 1u)] = SahSmall{root, (int)ci};
    }
    __syncthreads();
    for (;;) {
      __syncthreads();
      const int nb = S.nb;
      if (nb == 0) break;
      const SahNode en = S.bstack[nb - 1];
      const int b = en.b, e = en.e, side = en.sd & 1, depth = en.sd >> 1;
      const int plabel = en.parent;
      const bool is_root = plabel < 0;
      // centroid bounds
      float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
      for (int i = b + tid; i < e; i += kThreads) {
        const float4 c = __ldg(P.cen + ord[i]);
        mn[0] = fminf(mn[0], c.x); mn[1] = fminf(mn[1], c.y); mn[2] = fminf(mn[2], c.z);
        mx[0] = fmaxf(mx[0], c.x); mx[1] = fmaxf(mx[1], c.y); mx[2] = fmaxf(mx[2], c.z);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          mn[a] = fminf(mn[a], __shfl_xor_sync(FULL, mn[a], o));
          mx[a] = fmaxf(mx[a], __shfl_xor_sync(FULL, mx[a], o));
        }
      if (lane == 0)
        for (int a = 0; a < 3; ++a) { S.red[warp][a] = mn[a]; S.red[warp][3 + a] = mx[a]; }
      sah_clear_bins(S.bins, tid, kThreads);
      __syncthreads();
      if (tid < 6) {
        float v = S.red[0][tid];
        for (int w = 1; w < kWarps; ++w) v = tid < 3 ? fminf(v, S.red[w][tid]) : fmaxf(v, S.red[w][tid]);
        S.cb[tid] = v;
      }
      __syncthreads();
      float cb[6], scale[3];
#pragma unroll
      for (int k = 0; k < 6; ++k) cb[k] = S.cb[k];
#pragma unroll
      for (int a = 0; a < 3; ++a) scale[a] = cb[3 + a] > cb[a] ? (float)kSahBins / (cb[3 + a] - cb[a]) : 0.f;
      const bool median = depth >= kSahMaxDepth;
      if (!median)
        for (int i = b + tid; i < e; i += kThreads) sah_bin_prim(S.bins, P, ord[i], cb, scale);
      __syncthreads();
      if (warp == 0) {
        int axis = 0, kk = 0, nl = 0;
        if (!median) nl = sah_pick(S.bins, cb, lane, axis, kk);
        if (lane == 0) {
          S.m = nl > 0 ? b + nl : b + (e - b) / 2;
          S.axis = nl > 0 ? axis : -1;
          S.kk = kk;
        }
      }
      __syncthreads();
      const int m = S.m, axis = S.axis, kk = S.kk;
      if (axis >= 0) {
        // stable partition: block-wide ranks of the left flags, chunk by chunk
        int lbase = b, rbase = m;
        for (int i0 = b; i0 < e; i0 += kThreads) {
          const int i = i0 + tid;
          uint32_t p = 0;
          bool lft = false;
          if (i < e) {
            p = ord[i];
            lft = sah_bin(sah_c(__ldg(P.cen + p), axis), cb[axis], scale[axis]) < kk;
          }
          const unsigned bl = __ballot_sync(FULL, lft), br = __ballot_sync(FULL, i < e && !lft);
          __syncthreads();
          if (lane == 0) S.wsum[warp] = (uint32_t)__popc(bl) | ((uint32_t)__popc(br) << 16);
          __syncthreads();
          int lb = 0, rb = 0, lt = 0, rt = 0;
          for (int w = 0; w < kWarps; ++w) {
            const uint32_t v = S.wsum[w];
            if (w < warp) { lb += (int)(v & 0xffffu); rb += (int)(v >> 16); }
            lt += (int)(v & 0xffffu);
            rt += (int)(v >> 16);
          }
          const unsigned below = (1u << lane) - 1u;
          if (i < e) {
            if (lft) tmp[lbase + lb + __popc(bl & below)] = p;
            else tmp[rbase + rb + __popc(br & below)] = p;
          }
          lbase += lt;
          rbase += rt;
        }
        __syncthreads();
        for (int i = b + tid; i < e; i += kThreads) ord[i] = tmp[i];
      }
      __syncthreads();
      if (tid == 0) {
        --S.nb;
        if (is_root) {
          S.root_nat = f + m - 1 + shift;
          root_nat[ci] = S.root_nat;
        }
        const int label = sah_label(f, m, shift, R, S.root_nat, is_root);
        sah_emit(T, f, b, m, e, label, plabel, side, [&](int cb0, int ce0, int cs) {
          const SahNode ch{cb0, ce0, label, cs | ((depth + 1) << 1)};
          if (ce0 - cb0 > warp_max) S.bstack[S.nb++] = ch;
          else small[atomicAdd(nsmall, 1u)] = SahSmall{ch, (int)ci};
        });
      }
    }
    __syncthreads();
  }
}

constexpr int kSahSmallThreads = 128;

struct SahWarpSmem {
  uint32_t bins[kBinWords];
  SahNode stack[kSahWarpStack];
  // the triangles of a subtree of at most 32, one a lane: box corners (lo.w:
  // the bins per axis, 8 bits each), centroids (w: face id), and each lane's
  // best split
  float4 lo[32], hi[32], cen[32];
  float cost[32];
  int cand[32];  // candidate | left count << 8
};

// Builds the subtree of one node of 2..32 triangles, one triangle a lane, all
// its nodes of a level at once.  The splits are those of the binned search: a
// split after bin k keeps apart the same triangles as one after the highest
// occupied bin up to k, so each lane evaluates, per axis, the split after its
// own triangle's bin, over its node's triangles, and the node takes the
// lowest (cost, candidate).  Bound by its instructions, about 48 per
// (triangle, triangle) pair of a node; the bins of a warp-wide pass per node
// took ten times as many, half of them on nodes of 3 or 4 triangles.
__device__ __forceinline__ void sah_build32(SahWarpSmem& S, const SahTree& T, const SahPrims& P,
                                            uint32_t* __restrict__ ord, int f, int shift, int R, int& root_nat,
                                            const SahNode& en, int lane) {
  const unsigned FULL = 0xffffffffu;
  const int n = en.e - en.b;
  int s = 0, e = n, plabel = en.parent, side = en.sd & 1, depth = en.sd >> 1;
  uint32_t id = 0;
  if (lane < n) {
    id = ord[en.b + lane];
    float4 c = __ldg(P.cen + id);
    c.w = __uint_as_float(id);
    S.cen[lane] = c;
    S.lo[lane] = __ldg(P.lo + id);
    S.hi[lane] = __ldg(P.hi + id);
  } else {
    s = e = lane;  // no triangle: an empty node
  }
  __syncwarp();
  int longest = n;
  while (longest > 1) {
    const int len = e - s;
    float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
    int bin[3] = {0, 0, 0};
    bool flat[3] = {true, true, true};
    if (len > kSahTiny && depth < kSahMaxDepth) {
      // centroid bounds of the lane's node and the bins of its own centroid
      float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
      for (int j = s; j < e; ++j) {
        const float4 o = S.cen[j];
        mn[0] = fminf(mn[0], o.x); mn[1] = fminf(mn[1], o.y); mn[2] = fminf(mn[2], o.z);
        mx[0] = fmaxf(mx[0], o.x); mx[1] = fmaxf(mx[1], o.y); mx[2] = fmaxf(mx[2], o.z);
      }
      c = S.cen[lane];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        flat[a] = !(mx[a] > mn[a]);
        if (!flat[a]) bin[a] = sah_bin(sah_c(c, a), mn[a], (float)kSahBins / (mx[a] - mn[a]));
      }
      S.lo[lane].w = __int_as_float(bin[0] | (bin[1] << 8) | (bin[2] << 16));
    }
    __syncwarp();
    float cost = INFINITY;
    int cand = 0x7fffffff, nl = 0;
    if (len > kSahTiny && depth < kSahMaxDepth) {
      float l[3][6], r[3][6];
      int cl[3] = {0, 0, 0};
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          l[a][x] = r[a][x] = INFINITY;
          l[a][3 + x] = r[a][3 + x] = -INFINITY;
        }
      for (int j = s; j < e; ++j) {
        const float4 lo = S.lo[j], hi = S.hi[j];
        const int ob = __float_as_int(lo.w);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          if (((ob >> (8 * a)) & 0xff) <= bin[a]) {
            ++cl[a];
            l[a][0] = fminf(l[a][0], lo.x); l[a][1] = fminf(l[a][1], lo.y); l[a][2] = fminf(l[a][2], lo.z);
            l[a][3] = fmaxf(l[a][3], hi.x); l[a][4] = fmaxf(l[a][4], hi.y); l[a][5] = fmaxf(l[a][5], hi.z);
          } else {
            r[a][0] = fminf(r[a][0], lo.x); r[a][1] = fminf(r[a][1], lo.y); r[a][2] = fminf(r[a][2], lo.z);
            r[a][3] = fmaxf(r[a][3], hi.x); r[a][4] = fmaxf(r[a][4], hi.y); r[a][5] = fmaxf(r[a][5], hi.z);
          }
        }
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (flat[a] || cl[a] == len) continue;
        const float v = sah_half_area(l[a][0], l[a][1], l[a][2], l[a][3], l[a][4], l[a][5]) * (float)cl[a] +
                        sah_half_area(r[a][0], r[a][1], r[a][2], r[a][3], r[a][4], r[a][5]) * (float)(len - cl[a]);
        if (v < cost) {
          cost = v;
          cand = a * (kSahBins - 1) + bin[a];
          nl = cl[a];
        }
      }
    }
    S.cost[lane] = cost;
    S.cand[lane] = cand < 0x7fffffff ? (cand | (nl << 8)) : 0x7fffffff;
    __syncwarp();
    // the node's split: the lowest (cost, candidate) of its lanes
    int best = 0x7fffffff;
    if (len > kSahTiny && depth < kSahMaxDepth) {
      float bc = INFINITY;
      for (int j = s; j < e; ++j) {
        const float oc = S.cost[j];
        const int o = S.cand[j];
        if (oc < bc || (oc == bc && (o & 0xff) < (best & 0xff))) {
          bc = oc;
          best = o;
        }
      }
      if (!(bc < INFINITY)) best = 0x7fffffff;
    }
    bool left;
    int m;
    if (best != 0x7fffffff) {
      const int axis = (best & 0xff) / (kSahBins - 1), kk = (best & 0xff) % (kSahBins - 1);
      left = bin[axis == 0 ? 0 : (axis == 1 ? 1 : 2)] <= kk;
      m = s + (best >> 8);
    } else {
      m = s + len / 2;
      left = lane < m;
    }
    // stable partition: each triangle to its lane in the children's order
    const unsigned seg = len > 0 ? (0xffffffffu >> (32 - len)) << s : 0u;
    const unsigned lm = __ballot_sync(FULL, left) & seg;
    const unsigned below = (1u << lane) - 1u;
    const int to = left ? s + __popc(lm & below) : m + __popc(seg & ~lm & below);
    const float4 mylo = S.lo[lane], myhi = S.hi[lane], myc = S.cen[lane];
    __syncwarp();
    if (len > 1) {
      S.lo[to] = mylo;
      S.hi[to] = myhi;
      S.cen[to] = myc;
    }
    int label = 0;
    if (len > 1) {
      const bool is_root = plabel < 0;
      if (is_root) root_nat = f + en.b + m - 1 + shift;
      label = sah_label(f, en.b + m, shift, R, root_nat, is_root);
      if (lane == s)
        sah_emit(T, f, en.b + s, en.b + m, en.b + e, label, plabel, side, [](int, int, int) {});
      plabel = label;
      side = lane < m ? 0 : 1;
      ++depth;
      if (lane < m) e = m;
      else s = m;
    }
    __syncwarp();
    longest = __reduce_max_sync(FULL, e - s);
  }
  if (lane < n) ord[en.b + lane] = __float_as_uint(S.cen[lane].w);
  __syncwarp();
}

// One warp per node of the small list (grid-stride; the nodes' order in the
// list does not matter, each owns its range of the face order).
__global__ void __launch_bounds__(kSahSmallThreads)
    sah_small_kernel(const SahSmall* __restrict__ small, const uint32_t* __restrict__ nsmall,
                     const int32_t* __restrict__ clusters, const int32_t* __restrict__ root_nats, SahTree T,
                     uint32_t* __restrict__ order, uint32_t* __restrict__ tmp_all, SahPrims P) {
  pdl_wait();
  __shared__ SahWarpSmem smem[kSahSmallThreads / 32];
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  SahWarpSmem& S = smem[threadIdx.x >> 5];
  uint32_t* wb = S.bins;
  const uint32_t count = *nsmall, warps = gridDim.x * (kSahSmallThreads / 32);
  for (uint32_t si = blockIdx.x * (kSahSmallThreads / 32) + (threadIdx.x >> 5); si < count; si += warps) {
    const SahSmall it = small[si];
    const int R = clusters[it.cluster];
    // the cluster's range: a root of this list still has the radix tree's own
    // first and last; a split cluster's root was given the same ones
    const int f = T.first[R], l = T.last[R];
    const int shift = (R == l) ? 1 : 0;
    uint32_t* ord = order + f;
    uint32_t* tmp = tmp_all + f;
    int root_nat = it.node.parent < 0 ? 0 : root_nats[it.cluster];
    if (lane == 0) S.stack[0] = it.node;
    int sp = 1;
    __syncwarp();
    while (sp > 0) {
      const SahNode en = S.stack[sp - 1];
      --sp;
      __syncwarp();
      if (en.e - en.b <= 32) {
        sah_build32(S, T, P, ord, f, shift, R, root_nat, en, lane);
        continue;
      }
      const int b = en.b, e = en.e, side = en.sd & 1, depth = en.sd >> 1;
      const int plabel = en.parent;
      const bool is_root = plabel < 0;
      int m = b + (e - b) / 2;
      float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
      for (int i = b + lane; i < e; i += 32) {
        const float4 c = __ldg(P.cen + ord[i]);
        mn[0] = fminf(mn[0], c.x); mn[1] = fminf(mn[1], c.y); mn[2] = fminf(mn[2], c.z);
        mx[0] = fmaxf(mx[0], c.x); mx[1] = fmaxf(mx[1], c.y); mx[2] = fmaxf(mx[2], c.z);
      }
      float cb[6], scale[3];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          mn[a] = fminf(mn[a], __shfl_xor_sync(FULL, mn[a], o));
          mx[a] = fmaxf(mx[a], __shfl_xor_sync(FULL, mx[a], o));
        }
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        cb[a] = mn[a];
        cb[3 + a] = mx[a];
        scale[a] = mx[a] > mn[a] ? (float)kSahBins / (mx[a] - mn[a]) : 0.f;
      }
      int nl = 0, axis = 0, kk = 0;
      if (depth < kSahMaxDepth) {
        sah_clear_bins(wb, lane, 32);
        __syncwarp();
        for (int i = b + lane; i < e; i += 32) sah_bin_prim(wb, P, ord[i], cb, scale);
        __syncwarp();
        nl = sah_pick(wb, cb, lane, axis, kk);
        __syncwarp();
      }
      if (nl > 0) {
        m = b + nl;
        int lbase = b, rbase = m;
        for (int i0 = b; i0 < e; i0 += 32) {
          const int i = i0 + lane;
          uint32_t p = 0;
          bool lft = false;
          if (i < e) {
            p = ord[i];
            lft = sah_bin(sah_c(__ldg(P.cen + p), axis), cb[axis], scale[axis]) < kk;
          }
          const unsigned bl = __ballot_sync(FULL, lft), br = __ballot_sync(FULL, i < e && !lft);
          const unsigned below = (1u << lane) - 1u;
          if (i < e) {
            if (lft) tmp[lbase + __popc(bl & below)] = p;
            else tmp[rbase + __popc(br & below)] = p;
          }
          lbase += __popc(bl);
          rbase += __popc(br);
        }
        __syncwarp();
        for (int i = b + lane; i < e; i += 32) ord[i] = tmp[i];
        __syncwarp();
      }
      if (is_root) root_nat = f + m - 1 + shift;
      if (lane == 0) {
        const int label = sah_label(f, m, shift, R, root_nat, is_root);
        sah_emit(T, f, b, m, e, label, plabel, side, [&](int cb0, int ce0, int cs) {
          S.stack[sp++] = SahNode{cb0, ce0, label, cs | ((depth + 1) << 1)};
        });
      }
      sp = __shfl_sync(FULL, sp, 0);
      __syncwarp();
    }
  }
}

// clusters: internal nodes of 3..sah_max triangles whose parent has more (or
// that are a mesh root); sah_max <= kSahMax
__global__ void sah_find_kernel(const int64_t* __restrict__ face_off, int nmesh, int64_t n,
                                const int32_t* __restrict__ parent, const int32_t* __restrict__ first,
                                const int32_t* __restrict__ last, int sah_max, int32_t* __restrict__ clusters,
                                uint32_t* __restrict__ ncl) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int lo = 0, hi = nmesh - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (face_off[mid] <= i) lo = mid;
    else hi = mid - 1;
  }
  if (i >= face_off[lo + 1] - 1) return;  // the last position of a range has no internal node
  const int cnt = last[i] - first[i] + 1;
  if (cnt < 3 || cnt > sah_max) return;
  const int p = parent[i];
  if (p >= 0 && last[p] - first[p] + 1 <= sah_max) return;
  clusters[atomicAdd(ncl, 1u)] = (int32_t)i;
}

}  // namespace
}  // namespace a3d
