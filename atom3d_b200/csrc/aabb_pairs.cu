// MeshBVH.intersect_aabb modes 1-3: (box, face) pairs, optionally clipped.
//
// Replaces the pair output of bvh_aabb_intersect_kernel
// (atom3d/kernels/bvh_kernels.cu:555-610, host :1192-1242) and
// sat_clip_polygon_kernel / clip_with_plane (atom3d/kernels/cumtv_kernels.cu:
// 209-460) behind atom3d/core/mesh_bvh.py:297-479:
//   mode 1  every face passing SAT (sat_eps 1e-6) against the box
//   mode 2  those whose Sutherland-Hodgman clip against the box's 6 planes
//           (eps 1e-8) is non-empty, with the polygon's vertex count, its
//           centroid projected onto the triangle, and its fan area
//   mode 3  mode 2 plus the polygon's vertices (8 slots, zero padded)
//
// The tree walk finds the faces passing SAT and counts them per box, keeping
// each box's first eight; an exclusive scan of the counts gives each box its
// place, and a write pass copies the kept pairs there and walks the tree again
// for the boxes with more -- exact-size outputs, no truncation (the reference
// keeps at most min(100 N, 5e7) candidates and drops the rest silently).  Mode
// 1 writes the pairs directly.  Modes 2-3 write them as a candidate list (box,
// triangle slot) and clip it one thread per candidate: a flag pass (clip, hit
// mask), an exclusive scan of the flags, and an emit pass that clips the
// survivors again and writes the outputs at their compacted index.  (Clipping
// inside the divergent walk ran with one or two active lanes per warp and was
// 10x slower.)  Pairs come grouped by box in ascending order, in tree order
// within a box; the reference's order is that of an atomic counter.
//
// The clip is restated operation by operation with round-to-nearest
// intrinsics (IEEE divide and square root, no contraction), so the CPU
// oracle built with -ffp-contract=off reproduces it bit for bit.  An
// emitted vertex past the 8-slot polygon buffer is dropped (the reference
// writes it past its local array) and the count saturates at 8.
#include "box_query.cuh"
#include "primitives.cuh"

namespace a3d {
namespace {

constexpr int kClipMaxV = 8;
constexpr float kClipEps = 1e-8f;

// A polygon during the clip: its vertices' coordinates in the thread's column
// of shared memory, their order as a list of 4-bit slots in one register.  A
// plane that keeps all vertices costs their distances and a rotation of the
// list, a plane that cuts the polygon stores the new vertices alone (two,
// commonly): no vertex is copied and no array is indexed in local memory.
// Slots: at most 8 old vertices and 8 new ones are alive at a time.
// Bound by instruction issue (84% of the slots) at 13 of 32 lanes: the polygons
// of a warp have 0 to 7 vertices.  2.87M candidates (327,680 triangles in the
// voxels of a 512^3 grid): flag pass 476 -> 290 us, emit pass with polygons
// 613 -> 434 us against polygons in two local arrays copied at every plane.
constexpr int kClipThreads = 128;
constexpr int kClipSlots = 2 * kClipMaxV;
struct ClipSmem {
  float v[kClipSlots * 3][kClipThreads];
};

__device__ __forceinline__ float plane_dist(const float (*v)[kClipThreads], uint32_t slot, int axis, float sign,
                                            float d, bool full) {
  const uint32_t e = 3 * slot;
  const int t = threadIdx.x;
  if (!full) return fsb(fm(v[e + axis][t], sign), d);
  const float n0 = axis == 0 ? sign : 0.0f, n1 = axis == 1 ? sign : 0.0f, n2 = axis == 2 ? sign : 0.0f;
  return fsb(fa(fa(fm(v[e][t], n0), fm(v[e + 1][t], n1)), fm(v[e + 2][t], n2)), d);
}

// one clip step against n.p - d <= eps, n = sign * e_axis.  The products with
// the normal's zeros are left out where they cannot change the distance: full
// is set for coordinates that are not all finite, and a plane at 0 (where the
// sign of a zero distance could differ) takes them too.
__device__ __forceinline__ int clip_plane(float (*v)[kClipThreads], uint32_t& list, int n, int axis, float sign,
                                          float d, bool full) {
  const int t = threadIdx.x;
  full = full || d == 0.0f;
  unsigned in = 0, used = 0;
  for (int i = 0; i < n; ++i) {
    const uint32_t s = (list >> (4 * i)) & 15u;
    used |= 1u << s;
    if (plane_dist(v, s, axis, sign, d, full) <= kClipEps) in |= 1u << i;
  }
  const unsigned all = (1u << n) - 1u;
  if (in == 0u) return 0;
  if (in == all) {  // every vertex is kept, the second one first
    list = (list >> 4) | ((list & 15u) << (4 * (n - 1)));
    return n;
  }
  const unsigned qin = ((in >> 1) | (in << (n - 1))) & all;  // bit i: the end of edge i is inside
  unsigned todo = qin | (in ^ qin);
  uint32_t out = 0;
  int m = 0;
  while (todo && m < kClipMaxV) {
    const int i = __ffs((int)todo) - 1;
    todo &= todo - 1u;
    const uint32_t sp = (list >> (4 * i)) & 15u, sq = (list >> (4 * (i + 1 == n ? 0 : i + 1))) & 15u;
    if (((in ^ qin) >> i) & 1u) {
      const float dP = plane_dist(v, sp, axis, sign, d, full), dQ = plane_dist(v, sq, axis, sign, d, full);
      const float den = fsb(dP, dQ);
      if (fabsf(den) > kClipEps) {
        const float w = __fdiv_rn(dP, den);
        const uint32_t f = (uint32_t)__ffs((int)~used) - 1u;
        used |= 1u << f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const float x = v[3 * sp + a][t];
          v[3 * f + a][t] = fa(x, fm(w, fsb(v[3 * sq + a][t], x)));
        }
        out |= f << (4 * m);
        ++m;
      }
    }
    if (((qin >> i) & 1u) && m < kClipMaxV) {
      out |= sq << (4 * m);
      ++m;
    }
  }
  list = out;
  return m;
}

struct ClipOut {
  int count;
  float cx, cy, cz;  // centroid (projected onto the triangle)
  float area;
};

// Clips triangle t against the box; returns the vertex count (0 = empty).
// The polygon's vertices are in v, in the order of list.
__device__ __forceinline__ int clip_tri(const TriRec& t, const float mn[3], const float mx[3],
                                        float (*v)[kClipThreads], uint32_t& list) {
  const float p[9] = {t.a.x, t.a.y, t.a.z, t.b.x, t.b.y, t.b.z, t.c.x, t.c.y, t.c.z};
  bool full = false;  // a coordinate that is not finite, or whose differences may not be
#pragma unroll
  for (int e = 0; e < 9; ++e) {
    v[e][threadIdx.x] = p[e];
    full = full || !(fabsf(p[e]) < 1e37f);
  }
  list = 0x210u;
  int n = 3;
#pragma unroll
  for (int axis = 0; axis < 3; ++axis) {
    n = clip_plane(v, list, n, axis, 1.0f, mx[axis], full);
    if (!n) return 0;
    n = clip_plane(v, list, n, axis, -1.0f, -mn[axis], full);
    if (!n) return 0;
  }
  return n;
}

// centroid (mean clamped to the box, projected onto the triangle with
// clamped barycentrics) and fan area about the clamped mean
__device__ __forceinline__ ClipOut clip_measure(const TriRec& t, const float mn[3], const float mx[3],
                                                const float (*pv)[kClipThreads], uint32_t list, int cnt) {
  const int th = threadIdx.x;
  ClipOut o;
  o.count = cnt;
  o.area = 0.0f;
  float c[3] = {0.0f, 0.0f, 0.0f};
  for (int i = 0; i < cnt; ++i) {
    const uint32_t e = 3 * ((list >> (4 * i)) & 15u);
    c[0] = fa(c[0], pv[e][th]);
    c[1] = fa(c[1], pv[e + 1][th]);
    c[2] = fa(c[2], pv[e + 2][th]);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) c[a] = fminf(fmaxf(__fdiv_rn(c[a], (float)cnt), mn[a]), mx[a]);
  const float ax = t.a.x, ay = t.a.y, az = t.a.z, bx = t.b.x, by = t.b.y, bz = t.b.z;
  const float qx = t.c.x, qy = t.c.y, qz = t.c.z;
  const float e1x = fsb(bx, ax), e1y = fsb(by, ay), e1z = fsb(bz, az);
  const float e2x = fsb(qx, ax), e2y = fsb(qy, ay), e2z = fsb(qz, az);
  const float vx = fsb(c[0], ax), vy = fsb(c[1], ay), vz = fsb(c[2], az);
  const float d00 = dot3r(e1x, e1y, e1z, e1x, e1y, e1z);
  const float d01 = dot3r(e1x, e1y, e1z, e2x, e2y, e2z);
  const float d11 = dot3r(e2x, e2y, e2z, e2x, e2y, e2z);
  const float d20 = dot3r(vx, vy, vz, e1x, e1y, e1z);
  const float d21 = dot3r(vx, vy, vz, e2x, e2y, e2z);
  const float den = fsb(fm(d00, d11), fm(d01, d01));
  if (fabsf(den) < fm(kClipEps, kClipEps)) {
    o.cx = ax; o.cy = ay; o.cz = az;  // degenerate triangle: area stays 0
    return o;
  }
  float v = __fdiv_rn(fsb(fm(d11, d20), fm(d01, d21)), den);
  float w = __fdiv_rn(fsb(fm(d00, d21), fm(d01, d20)), den);
  float u = fsb(fsb(1.0f, v), w);
  if (u < 0.0f) u = 0.0f;
  if (v < 0.0f) v = 0.0f;
  if (w < 0.0f) w = 0.0f;
  float nn = fa(fa(u, v), w);
  if (nn <= kClipEps) { u = 1.0f; v = 0.0f; w = 0.0f; nn = 1.0f; }
  u = __fdiv_rn(u, nn); v = __fdiv_rn(v, nn); w = __fdiv_rn(w, nn);
  o.cx = fa(fa(fm(u, ax), fm(v, bx)), fm(w, qx));
  o.cy = fa(fa(fm(u, ay), fm(v, by)), fm(w, qy));
  o.cz = fa(fa(fm(u, az), fm(v, bz)), fm(w, qz));
  float ar = 0.0f;
  uint32_t e = 3 * (list & 15u);
  const float f0 = fsb(pv[e][th], c[0]), f1 = fsb(pv[e + 1][th], c[1]), f2 = fsb(pv[e + 2][th], c[2]);
  float p0 = f0, p1 = f1, p2 = f2;
  for (int i = 1; i <= cnt; ++i) {
    float q0 = f0, q1 = f1, q2 = f2;
    if (i < cnt) {
      e = 3 * ((list >> (4 * i)) & 15u);
      q0 = fsb(pv[e][th], c[0]); q1 = fsb(pv[e + 1][th], c[1]); q2 = fsb(pv[e + 2][th], c[2]);
    }
    const float x = fsb(fm(p1, q2), fm(p2, q1)), y = fsb(fm(p2, q0), fm(p0, q2)), z = fsb(fm(p0, q1), fm(p1, q0));
    ar = fa(ar, fm(0.5f, __fsqrt_rn(dot3r(x, y, z, x, y, z))));
    p0 = q0; p1 = q1; p2 = q2;
  }
  o.area = ar < kClipEps ? 0.0f : ar;
  return o;
}

struct PairOut {
  void* aabb_ids;  // int32 (mode 1) or int64 (modes 2-3)
  void* face_ids;
  int32_t* poly_counts;
  float* centroids;
  float* areas;
  float* poly_verts;  // mode 3
};

// Clips candidate k (box cand_box[k], triangle record cand_slot[k]).
template <bool kEmit, int kMode>
__device__ __forceinline__ void clip_candidate(const TriRec* __restrict__ tris, const float* __restrict__ bmin,
                                               const float* __restrict__ bmax, const uint32_t* __restrict__ cand_box,
                                               const uint32_t* __restrict__ cand_slot, int64_t k,
                                               uint32_t* __restrict__ flags, uint8_t* __restrict__ hit,
                                               const int64_t* __restrict__ coffs, const PairOut& out,
                                               int64_t n, int64_t num_slots, int64_t num_pairs,
                                               unsigned long long* __restrict__ faults, ClipSmem& S) {
  if (kEmit && !flags[k]) return;
  const int64_t i = cand_box[k];
  const uint32_t slot = cand_slot[k];
  if (i >= n || slot >= num_slots) {  // never for a candidate list written by the walk
    atomicAdd(faults, 1ull);
    if (!kEmit) flags[k] = 0;
    return;
  }
  const float4* p = reinterpret_cast<const float4*>(tris + slot);
  TriRec t;
  t.a = __ldg(p); t.b = __ldg(p + 1); t.c = __ldg(p + 2); t.r = make_float4(0.f, 0.f, 0.f, 0.f);
  const float mn[3] = {bmin[3 * i], bmin[3 * i + 1], bmin[3 * i + 2]};
  const float mx[3] = {bmax[3 * i], bmax[3 * i + 1], bmax[3 * i + 2]};
  uint32_t list;
  const int cnt = clip_tri(t, mn, mx, S.v, list);
  if (!kEmit) {
    flags[k] = cnt > 0;
    if (cnt > 0) hit[i] = 1;
    return;
  }
  const int64_t o = coffs[k];
  if (!cnt || o < 0 || o >= num_pairs) {  // the flag pass decided this clip differently
    atomicAdd(faults, 1ull);
    return;
  }
  const ClipOut c = clip_measure(t, mn, mx, S.v, list, cnt);
  reinterpret_cast<int64_t*>(out.aabb_ids)[o] = i;
  reinterpret_cast<int64_t*>(out.face_ids)[o] = __float_as_int(t.a.w);
  out.poly_counts[o] = c.count;
  out.centroids[3 * o] = c.cx;
  out.centroids[3 * o + 1] = c.cy;
  out.centroids[3 * o + 2] = c.cz;
  out.areas[o] = c.area;
  if (kMode == 3) {
    float4* pv = reinterpret_cast<float4*>(out.poly_verts + 24 * o);
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      float e[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int f = 4 * q + u, vi = f / 3, ax = f % 3;
        e[u] = vi < cnt ? S.v[3 * ((list >> (4 * vi)) & 15u) + ax][threadIdx.x] : 0.0f;
      }
      pv[q] = make_float4(e[0], e[1], e[2], e[3]);
    }
  }
}

__global__ void __launch_bounds__(kClipThreads)
    clip_flags_kernel(const TriRec* __restrict__ tris, const float* __restrict__ bmin,
                                  const float* __restrict__ bmax, const uint32_t* __restrict__ cand_box,
                                  const uint32_t* __restrict__ cand_slot, int64_t m, uint32_t* __restrict__ flags,
                                  uint8_t* __restrict__ hit, int64_t n, int64_t num_slots,
                                  unsigned long long* __restrict__ faults) {
  pdl_wait();
  __shared__ ClipSmem S;
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m)
    clip_candidate<false, 2>(tris, bmin, bmax, cand_box, cand_slot, k, flags, hit, nullptr, PairOut{}, n, num_slots,
                             0, faults, S);
}

template <int kMode>
__global__ void __launch_bounds__(kClipThreads)
    clip_emit_kernel(const TriRec* __restrict__ tris, const float* __restrict__ bmin,
                                 const float* __restrict__ bmax, const uint32_t* __restrict__ cand_box,
                                 const uint32_t* __restrict__ cand_slot, int64_t m, uint32_t* __restrict__ flags,
                                 const int64_t* __restrict__ coffs, PairOut out, int64_t n, int64_t num_slots,
                                 unsigned long long* __restrict__ faults) {
  pdl_wait();
  __shared__ ClipSmem S;
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m)
    clip_candidate<true, kMode>(tris, bmin, bmax, cand_box, cand_slot, k, flags, nullptr, coffs, out, n, num_slots,
                                coffs[m], faults, S);
}

// The count pass keeps each box's first kPairsKept pairs, one 32-byte sector:
// the write pass copies them, and walks the tree again only for the boxes with
// more (listed by the count pass): 20 + 66 us for 933,270 voxels of 3.07 pairs
// each, against 450 us for walking all of them again.
constexpr int kPairsKept = 8;

// Writes box i's pair at o: the face (kSlots false) or the triangle record.
template <bool kSlots>
__device__ __forceinline__ void put_pair(const TriRec* __restrict__ tris, int64_t num_slots, int64_t i, uint32_t slot,
                                         int64_t o, int64_t end, int32_t* __restrict__ out_box,
                                         int32_t* __restrict__ out_face, unsigned long long* __restrict__ faults) {
  if (o >= end || slot >= num_slots) {  // never: the count pass found the same pairs
    atomicAdd(faults, 1ull);
    return;
  }
  out_box[o] = (int32_t)i;
  out_face[o] = kSlots ? (int32_t)slot : __float_as_int(__ldg(&tris[slot].a.w));
}

struct PairsWs {
  uint32_t* counts;
  int64_t* offs;
  int64_t* scan_tmp;
  uint32_t* kept;   // [n][kPairsKept] triangle records
  uint32_t* longs;  // boxes with more pairs than are kept
  unsigned long long* misc;  // [0] overflow, [1] guard faults, [2] boxes in longs
};

size_t carve_pairs(PairsWs& w, Workspace& ws, int64_t n) {
  w.counts = ws.take<uint32_t>(n);
  w.offs = ws.take<int64_t>(n + 1);
  w.scan_tmp = ws.take<int64_t>((int64_t)scan_workspace_elems(n));
  w.kept = ws.take<uint32_t>(n * kPairsKept);
  w.longs = ws.take<uint32_t>(n);
  w.misc = ws.take<unsigned long long>(3);
  return ws.used;
}

struct ClipWs {
  uint32_t* cand_box;
  uint32_t* cand_slot;
  uint32_t* flags;
  int64_t* coffs;
  int64_t* scan_tmp;
};

size_t carve_clip(ClipWs& w, Workspace& ws, int64_t m) {
  w.cand_box = ws.take<uint32_t>(m);
  w.cand_slot = ws.take<uint32_t>(m);
  w.flags = ws.take<uint32_t>(m);
  w.coffs = ws.take<int64_t>(m + 1);
  w.scan_tmp = ws.take<int64_t>((int64_t)scan_workspace_elems(m));
  return ws.used;
}

__device__ __forceinline__ void load_box(const float* __restrict__ bmin, const float* __restrict__ bmax, int64_t i,
                                         float* mn, float* mx) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    mn[a] = bmin[3 * i + a];
    mx[a] = bmax[3 * i + a];
  }
}

struct CountQuery {
  const float* bmin;
  const float* bmax;
  uint32_t* counts;
  uint8_t* hit;
  uint32_t* kept;
  uint32_t* longs;
  unsigned long long* misc;
  uint32_t i = 0, c = 0;
  __device__ __forceinline__ void begin(int64_t k, float* mn, float* mx) {
    i = (uint32_t)k;
    c = 0;
    load_box(bmin, bmax, k, mn, mx);
  }
  __device__ __forceinline__ void leaf(uint32_t mask, uint32_t first) {
    for (uint32_t m = mask; m && c < (uint32_t)kPairsKept; m &= m - 1u) {
      kept[(int64_t)kPairsKept * i + c] = first + (uint32_t)__ffs((int)m) - 1u;
      ++c;
      mask &= mask - 1u;
    }
    c += (uint32_t)__popc(mask);
  }
  __device__ __forceinline__ void done(bool overflow) {
    if (overflow) atomicExch(misc, 1ull);
    if (c > (uint32_t)kPairsKept) longs[atomicAdd(misc + 2, 1ull)] = i;
    counts[i] = c;
    if (hit) hit[i] = c > 0;
  }
};

__global__ void __launch_bounds__(kBoxThreads, kBoxBlocks)
    pairs_count_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris, int64_t n, int64_t per,
                       CountQuery query) {
  pdl_wait();
  __shared__ BoxSmem smem[kBoxWarps];
  const int64_t pos = ((int64_t)blockIdx.x * kBoxWarps + (threadIdx.x >> 5)) * per;
  CountQuery q = query;
  box_walk(nodes, tris, pos, pos + per < n ? pos + per : n, smem[threadIdx.x >> 5], q);
}

// the boxes whose pairs were all kept, one a thread
template <bool kSlots>
__global__ void pairs_copy_kernel(const TriRec* __restrict__ tris, int64_t num_slots, int64_t n, PairsWs w,
                                  int32_t* __restrict__ out_box, int32_t* __restrict__ out_face) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t c = w.counts[i];
  if (c == 0 || c > (uint32_t)kPairsKept) return;
  const int64_t o = w.offs[i], end = w.offs[i + 1];
  const uint4 lo = *reinterpret_cast<const uint4*>(w.kept + kPairsKept * i);
  uint4 hi = make_uint4(0, 0, 0, 0);
  if (c > 4) hi = *reinterpret_cast<const uint4*>(w.kept + kPairsKept * i + 4);
  const uint32_t r[kPairsKept] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
  for (int k = 0; k < kPairsKept; ++k)
    if (k < (int)c) put_pair<kSlots>(tris, num_slots, i, r[k], o + k, end, out_box, out_face, w.misc + 1);
}

template <bool kSlots>
struct WriteQuery {
  const float* bmin;
  const float* bmax;
  const TriRec* tris;
  int64_t num_slots;
  PairsWs w;
  int32_t* out_box;
  int32_t* out_face;
  uint32_t i = 0;
  int64_t o = 0, end = 0;
  __device__ __forceinline__ void begin(int64_t k, float* mn, float* mx) {
    i = w.longs[k];
    o = w.offs[i];
    end = w.offs[i + 1];
    load_box(bmin, bmax, i, mn, mx);
  }
  __device__ __forceinline__ void leaf(uint32_t mask, uint32_t first) {
    for (; mask; mask &= mask - 1u)
      put_pair<kSlots>(tris, num_slots, i, first + (uint32_t)__ffs((int)mask) - 1u, o++, end, out_box, out_face,
                       w.misc + 1);
  }
  __device__ __forceinline__ void done(bool) {}
};

// the boxes with more pairs than were kept: the walk again
template <bool kSlots>
__global__ void __launch_bounds__(kBoxThreads, kBoxBlocks)
    pairs_write_kernel(const WideNode* __restrict__ nodes, WriteQuery<kSlots> query) {
  pdl_wait();
  __shared__ BoxSmem smem[kBoxWarps];
  WriteQuery<kSlots> q = query;
  box_walk_all(nodes, q.tris, (int64_t)q.w.misc[2], smem[threadIdx.x >> 5], q);
}

template <bool kSlots>
int launch_write(const a3d_bvh_view* bvh, const float* bmin, const float* bmax, int64_t n, const PairsWs& w,
                 int32_t* out_box, int32_t* out_face, cudaStream_t s) {
  const WideNode* nodes = (const WideNode*)bvh->nodes;
  const TriRec* tris = (const TriRec*)bvh->tris;
  const WriteQuery<kSlots> q{bmin, bmax, tris, bvh->num_tris, w, out_box, out_face};
  A3D_PDL(pairs_copy_kernel<kSlots>, dim3((unsigned)ceil_div(n, 256)), dim3(256), 0, s, tris, bvh->num_tris, n, w,
          out_box, out_face);
  A3D_PDL(pairs_write_kernel<kSlots>, dim3((unsigned)box_blocks(n, num_sms())), dim3(kBoxThreads), 0, s, nodes, q);
  return A3D_OK;
}

}  // namespace
}  // namespace a3d

using namespace a3d;

extern "C" size_t a3d_aabb_pairs_workspace_bytes(int64_t n) {
  Workspace ws(nullptr, 0);
  PairsWs w;
  return carve_pairs(w, ws, n > 0 ? n : 1) + 256;
}

extern "C" size_t a3d_aabb_clip_workspace_bytes(int64_t num_candidates) {
  Workspace ws(nullptr, 0);
  ClipWs w;
  return carve_clip(w, ws, num_candidates > 0 ? num_candidates : 1) + 256;
}

namespace {
int check_pairs_args(const a3d_bvh_view* bvh, int mode, int64_t n) {
  A3D_REQUIRE(bvh && bvh->nodes && bvh->tris, A3D_ERR_ARGUMENT, "aabb_pairs: invalid bvh");
  A3D_REQUIRE(mode >= 1 && mode <= 3, A3D_ERR_ARGUMENT, "aabb_pairs: mode must be 1, 2 or 3");
  A3D_REQUIRE(n >= 0 && n < (1ll << 31), A3D_ERR_ARGUMENT, "aabb_pairs: bad size");
  return A3D_OK;
}
}  // namespace

extern "C" int a3d_aabb_pairs_count(const a3d_bvh_view* bvh, const float* box_min, const float* box_max, int64_t n,
                                    int mode, uint8_t* hit, void* workspace, size_t workspace_bytes,
                                    int64_t* num_candidates_out, a3d_stream_t stream) {
  cudaStream_t s = (cudaStream_t)stream;
  A3D_TRY(check_pairs_args(bvh, mode, n));
  A3D_REQUIRE(num_candidates_out, A3D_ERR_ARGUMENT, "aabb_pairs: null count output");
  *num_candidates_out = 0;
  if (n == 0) return A3D_OK;
  A3D_REQUIRE(box_min && box_max && hit, A3D_ERR_ARGUMENT, "aabb_pairs: null pointer");
  Workspace ws(workspace, workspace_bytes);
  PairsWs w;
  carve_pairs(w, ws, n);
  A3D_REQUIRE(workspace && ws.ok(), A3D_ERR_WORKSPACE, "aabb_pairs: workspace too small");
  A3D_CUDA_TRY(cudaMemsetAsync(w.misc, 0, 3 * sizeof(unsigned long long), s));
  // modes 2-3: the hit mask comes from the clip
  uint8_t* h = mode == 1 ? hit : nullptr;
  const WideNode* nodes = (const WideNode*)bvh->nodes;
  const TriRec* tris = (const TriRec*)bvh->tris;
  const int64_t per = box_items(n, (int64_t)num_sms() * kBoxBlocks * kBoxWarps);
  const CountQuery q{box_min, box_max, w.counts, h, w.kept, w.longs, w.misc};
  A3D_PDL(pairs_count_kernel, dim3((unsigned)ceil_div(n, per * kBoxWarps)), dim3(kBoxThreads), 0, s, nodes, tris, n,
          per, q);
  A3D_TRY((device_exclusive_scan<uint32_t, int64_t>(w.counts, w.offs, n, w.scan_tmp, w.offs + n, s)));
  unsigned long long misc[3];
  int64_t total = 0;
  A3D_CUDA_TRY(cudaMemcpyAsync(misc, w.misc, sizeof(misc), cudaMemcpyDeviceToHost, s));
  A3D_CUDA_TRY(cudaMemcpyAsync(&total, w.offs + n, sizeof(total), cudaMemcpyDeviceToHost, s));
  A3D_CUDA_TRY(cudaStreamSynchronize(s));
  A3D_REQUIRE(misc[0] == 0, A3D_ERR_OVERFLOW, "aabb_pairs: traversal stack overflow");
  *num_candidates_out = total;
  return A3D_OK;
}

extern "C" int a3d_aabb_pairs_clip(const a3d_bvh_view* bvh, const float* box_min, const float* box_max, int64_t n,
                                   void* workspace, size_t workspace_bytes, void* clip_workspace,
                                   size_t clip_workspace_bytes, int64_t num_candidates, uint8_t* hit,
                                   int64_t* num_pairs_out, a3d_stream_t stream) {
  cudaStream_t s = (cudaStream_t)stream;
  A3D_TRY(check_pairs_args(bvh, 2, n));
  A3D_REQUIRE(num_pairs_out && num_candidates >= 0 && num_candidates < (1ll << 32), A3D_ERR_ARGUMENT,
              "aabb_pairs_clip: bad argument");
  *num_pairs_out = 0;
  if (n == 0) return A3D_OK;
  A3D_REQUIRE(box_min && box_max && hit, A3D_ERR_ARGUMENT, "aabb_pairs_clip: null pointer");
  Workspace ws(workspace, workspace_bytes);
  PairsWs w;
  carve_pairs(w, ws, n);
  Workspace cws(clip_workspace, clip_workspace_bytes);
  ClipWs c;
  carve_clip(c, cws, num_candidates);
  A3D_REQUIRE(workspace && ws.ok() && clip_workspace && cws.ok(), A3D_ERR_WORKSPACE,
              "aabb_pairs_clip: workspace too small");
  A3D_CUDA_TRY(cudaMemsetAsync(hit, 0, n, s));
  if (num_candidates == 0) return A3D_OK;
  A3D_TRY(launch_write<true>(bvh, box_min, box_max, n, w, (int32_t*)c.cand_box, (int32_t*)c.cand_slot, s));
  A3D_PDL(clip_flags_kernel, dim3((unsigned)ceil_div(num_candidates, kClipThreads)), dim3(kClipThreads), 0, s, (const TriRec*)bvh->tris,
          box_min, box_max, c.cand_box, c.cand_slot, num_candidates, c.flags, hit, n, bvh->num_tris, w.misc + 1);
  A3D_TRY((device_exclusive_scan<uint32_t, int64_t>(c.flags, c.coffs, num_candidates, c.scan_tmp,
                                                     c.coffs + num_candidates, s)));
  int64_t total = 0;
  unsigned long long faults = 0;
  A3D_CUDA_TRY(cudaMemcpyAsync(&total, c.coffs + num_candidates, sizeof(total), cudaMemcpyDeviceToHost, s));
  A3D_CUDA_TRY(cudaMemcpyAsync(&faults, w.misc + 1, sizeof(faults), cudaMemcpyDeviceToHost, s));
  A3D_CUDA_TRY(cudaStreamSynchronize(s));
  A3D_REQUIRE(faults == 0, A3D_ERR_OVERFLOW, "aabb_pairs_clip: a candidate index guard fired");
  *num_pairs_out = total;
  return A3D_OK;
}

extern "C" int a3d_aabb_pairs_write(const a3d_bvh_view* bvh, const float* box_min, const float* box_max, int64_t n,
                                    int mode, void* workspace, size_t workspace_bytes, void* clip_workspace,
                                    size_t clip_workspace_bytes, int64_t num_candidates, void* aabb_ids,
                                    void* face_ids, int32_t* poly_counts, float* centroids, float* areas,
                                    float* poly_verts, a3d_stream_t stream) {
  cudaStream_t s = (cudaStream_t)stream;
  A3D_TRY(check_pairs_args(bvh, mode, n));
  if (n == 0) return A3D_OK;
  A3D_REQUIRE(box_min && box_max && aabb_ids && face_ids, A3D_ERR_ARGUMENT, "aabb_pairs: null output");
  Workspace ws(workspace, workspace_bytes);
  PairsWs w;
  carve_pairs(w, ws, n);
  A3D_REQUIRE(workspace && ws.ok(), A3D_ERR_WORKSPACE, "aabb_pairs: workspace too small");
  if (mode == 1) {
    A3D_TRY(launch_write<false>(bvh, box_min, box_max, n, w, (int32_t*)aabb_ids, (int32_t*)face_ids, s));
  } else {
    A3D_REQUIRE(poly_counts && centroids && areas, A3D_ERR_ARGUMENT, "aabb_pairs: null clip output");
    A3D_REQUIRE(mode != 3 || (poly_verts && ((uintptr_t)poly_verts & 15) == 0), A3D_ERR_ARGUMENT,
                "aabb_pairs: poly_verts must be a 16-byte aligned [P,8,3] buffer");
    Workspace cws(clip_workspace, clip_workspace_bytes);
    ClipWs c;
    carve_clip(c, cws, num_candidates);
    A3D_REQUIRE(clip_workspace && cws.ok() && num_candidates >= 0, A3D_ERR_WORKSPACE,
                "aabb_pairs: clip workspace too small");
    if (num_candidates == 0) return A3D_OK;
    const PairOut out{aabb_ids, face_ids, poly_counts, centroids, areas, poly_verts};
    const unsigned g = (unsigned)ceil_div(num_candidates, kClipThreads);
    if (mode == 2)
      A3D_PDL(clip_emit_kernel<2>, dim3(g), dim3(kClipThreads), 0, s, (const TriRec*)bvh->tris, box_min, box_max, c.cand_box,
              c.cand_slot, num_candidates, c.flags, c.coffs, out, n, bvh->num_tris, w.misc + 1);
    else
      A3D_PDL(clip_emit_kernel<3>, dim3(g), dim3(kClipThreads), 0, s, (const TriRec*)bvh->tris, box_min, box_max, c.cand_box,
              c.cand_slot, num_candidates, c.flags, c.coffs, out, n, bvh->num_tris, w.misc + 1);
  }
  unsigned long long faults = 0;
  A3D_CUDA_TRY(cudaMemcpyAsync(&faults, w.misc + 1, sizeof(faults), cudaMemcpyDeviceToHost, s));
  A3D_CUDA_TRY(cudaStreamSynchronize(s));
  A3D_REQUIRE(faults == 0, A3D_ERR_OVERFLOW, "aabb_pairs_write: an output index guard fired");
  return A3D_OK;
}
