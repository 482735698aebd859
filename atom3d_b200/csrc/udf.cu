// Closest-triangle queries over the wide BVH: UDF, fused pseudo-normal SDF
// sign, learned-bound seeding, and the distance adjoints.
//
// Replaces bvh_udf_kernel (atom3d/kernels/bvh_kernels.cu:363-463) and the
// PyTorch sign gathers of MeshBVH._compute_sign (atom3d/core/mesh_bvh.py:
// 759-827).  Design:
//   * many queries are Morton-sorted (in-house radix sort) so a warp walks
//     neighbouring regions of the tree together;
//   * a group of four or two lanes walks the tree for one query: each lane
//     tests one or two of a node's children, first the box, then the disc
//     about the child's triangles (bvh_children.cuh); the nearest qualifying
//     child by box distance is visited next and the others pushed;
//   * the traversal stack lives in shared memory and continues in the
//     workspace; a query that would overflow both is re-run by a launch with a
//     deep local-memory stack, never truncated;
//   * a per-query bound (learned upper bound on the distance) seeds the
//     pruning radius; a query whose bound proves too small is run again
//     without it, so results are identical with and without the bound;
//   * the traversal leaves (triangle, squared distance) per query, and a
//     second kernel makes the closest point, barycentrics and sign of them.
#include <math.h>

#include "bvh_layout.cuh"
#include "bvh_children.cuh"
#include "primitives.cuh"
#include "tri_math.cuh"

namespace a3d {

namespace {

constexpr int kUdfThreads = 128;
constexpr int kSharedDepth = 32;
constexpr int kDeepDepth = 256;

struct SignArgs {
  const float* face_normals;
  const float* vertex_pn;
  const float* edge_pn;
  const int64_t* he_edge_idx;
  const int32_t* faces;
};

struct QueryOut {
  float* dist;
  int32_t* fid;
  float* cp;
  float* uvw;
};

// the traversals' results, in the caller's order of the queries: closest
// triangle (0xffffffff: none) and squared distance, turned into the caller's
// outputs by udf_finish_kernel
struct Best {
  uint32_t* tri;
  float* sq;
};

struct Counters {
  unsigned long long nodes;
  unsigned long long tris;
};

// Which tree a query walks.  One mesh: the root is node 0.  A batch: query
// qi (index qbase + qi in the caller's array) belongs to mesh m with
// qoff[m] <= qbase + qi < qoff[m+1], whose root is roots[m].
struct MeshSel {
  const int64_t* qoff;
  const uint32_t* roots;
  int nmesh;
  int64_t qbase;
  __device__ __forceinline__ uint32_t root_of(int64_t qi) const {
    if (qoff == nullptr) return 0u;
    const int64_t g = qbase + qi;
    int lo = 0, hi = nmesh - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(qoff + mid) <= g) lo = mid;
      else hi = mid - 1;
    }
    return __ldg(roots + lo);
  }
};

// children are visited in ascending (distance, ref) order: a total order, so
// every traversal variant (single lane, quad of lanes) walks the same
// sequence and breaks distance ties identically
__device__ __forceinline__ bool child_less(float da, uint32_t ra, float db, uint32_t rb) {
  return da < db || (da == db && ra < rb);
}

__device__ __forceinline__ void cswap(float& da, uint32_t& ra, float& db, uint32_t& rb) {
  if (child_less(db, rb, da, ra)) {
    float t = da; da = db; db = t;
    uint32_t u = ra; ra = rb; rb = u;
  }
}

__device__ __forceinline__ float box_dist_sq(float px, float py, float pz, float lx, float ly, float lz, float hx,
                                             float hy, float hz) {
  const float dx = fmaxf(fmaxf(lx - px, px - hx), 0.f);
  const float dy = fmaxf(fmaxf(ly - py, py - hy), 0.f);
  const float dz = fmaxf(fmaxf(lz - pz, pz - hz), 0.f);
  return dx * dx + dy * dy + dz * dz;
}

// FP64 evaluation for near-degenerate triangles, kept out of line so the
// hot loop does not carry its registers.
__device__ __noinline__ float tri_dist_sq_f64(float ax, float ay, float az, float bx, float by, float bz, float cx,
                                              float cy, float cz, float px, float py, float pz) {
  const double d = TriEval<double>::dist_sq(mk<double>(px, py, pz), mk<double>(ax, ay, az), mk<double>(bx, by, bz),
                                            mk<double>(cx, cy, cz));
  return (float)d;
}

__device__ __forceinline__ float tri_dist_sq(const TriRec& t, float px, float py, float pz) {
  if (t.c.w < 0.f)  // near-degenerate
    return tri_dist_sq_f64(t.a.x, t.a.y, t.a.z, t.b.x, t.b.y, t.b.z, t.c.x, t.c.y, t.c.z, px, py, pz);
  return dist_sq_bary(mk(px, py, pz), mk(t.a.x, t.a.y, t.a.z), mk(t.b.x, t.b.y, t.b.z), mk(t.c.x, t.c.y, t.c.z),
                      t.c.w, t.b.w, t.r.w, t.r.x, t.r.y, t.r.z);
}

__device__ __forceinline__ TriRec load_tri(const TriRec* tris, uint32_t i) {
  const float4* p = reinterpret_cast<const float4*>(tris + i);
  TriRec r;
  r.a = __ldg(p);
  r.b = __ldg(p + 1);
  r.c = __ldg(p + 2);
  r.r = __ldg(p + 3);
  return r;
}

// The arrays a traversal reads.  With kGuard (batches, whose node count is
// only known on the device) a node or triangle index outside the arrays is
// recorded in *fault (kFaultNode / kFaultTri) and replaced by 0, so no
// access leaves them whatever the tree holds.  The child records hold no
// reference outside the arrays (child_kernel): a bad one is there the leaf at
// num_tris, which has a disc of its own and is recorded by the triangle read.
constexpr uint32_t kFaultNode = 1u, kFaultTri = 2u;

template <bool kGuard>
struct TreeT {
  const WideNode* __restrict__ nodes;
  const TriRec* __restrict__ tris;
  uint32_t num_nodes;
  uint32_t num_tris;
  uint32_t* fault;
  ChildRecs children;
  uint32_t num_children;  // a node past them has no records (0: none at all)
  __device__ __forceinline__ const int4* node(uint32_t ref) const {
    if (kGuard && ref >= num_nodes) {
      atomicOr(fault, kFaultNode);
      ref = 0;
    }
    return reinterpret_cast<const int4*>(nodes + ref);
  }
  __device__ __forceinline__ TriRec tri(uint32_t i) const {
    if (kGuard && i >= num_tris) {
      atomicOr(fault, kFaultTri);
      i = 0;
    }
    return load_tri(tris, i);
  }
};

// Stack in shared memory, [depth][blockDim] layout.
struct SharedStack {
  uint2* base;  // points at s[0][threadIdx.x]
  int sp;
  static constexpr int kDepth = kSharedDepth;
  __device__ __forceinline__ void push(uint32_t ref, float d) {
    base[sp * kUdfThreads] = make_uint2(ref, __float_as_uint(d));
    ++sp;
  }
  __device__ __forceinline__ uint2 pop() {
    --sp;
    return base[sp * kUdfThreads];
  }
};

struct LocalStack {
  uint2 s[kDeepDepth];
  int sp;
  static constexpr int kDepth = kDeepDepth;
  __device__ __forceinline__ void push(uint32_t ref, float d) { s[sp++] = make_uint2(ref, __float_as_uint(d)); }
  __device__ __forceinline__ uint2 pop() { return s[--sp]; }
};

// Core traversal.  Returns false when the stack would overflow (result then
// invalid).  best_sq: in = initial pruning radius^2, out = best distance^2.
template <typename Stack, typename Tree>
__device__ __forceinline__ bool traverse(const Tree& T, float px, float py, float pz, Stack& st, float& best_sq,
                                         uint32_t& best_tri, Counters& ctr, uint32_t root = 0u) {
  uint32_t ref = root;  // a root is always an internal node (a single-leaf tree still has one)
  bool have = true;
  for (;;) {
    if (have) {
      if (!ref_is_leaf(ref)) {
        ++ctr.nodes;
        const int4* np = T.node(ref);
        const int4 w0 = __ldg(np), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3);
        const float ox = __int_as_float(w0.x), oy = __int_as_float(w0.y), oz = __int_as_float(w0.z);
        const uint32_t meta = (uint32_t)w0.w;
        const float sx = __uint_as_float((meta & 0xffu) << 23);
        const float sy = __uint_as_float(((meta >> 8) & 0xffu) << 23);
        const float sz = __uint_as_float(((meta >> 16) & 0xffu) << 23);
        const uint32_t qlx = (uint32_t)w1.x, qly = (uint32_t)w1.y, qlz = (uint32_t)w1.z;
        const uint32_t qhx = (uint32_t)w1.w, qhy = (uint32_t)w2.x, qhz = (uint32_t)w2.y;
        float d[4];
        uint32_t r[4] = {(uint32_t)w2.z, (uint32_t)w2.w, (uint32_t)w3.x, (uint32_t)w3.y};
        const int nch = (int)(meta >> 24);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float lx = dequant(qlx, c, sx, ox);
          const float ly = dequant(qly, c, sy, oy);
          const float lz = dequant(qlz, c, sz, oz);
          const float hx = dequant(qhx, c, sx, ox);
          const float hy = dequant(qhy, c, sy, oy);
          const float hz = dequant(qhz, c, sz, oz);
          d[c] = c < nch ? box_dist_sq(px, py, pz, lx, ly, lz, hx, hy, hz) : INFINITY;
        }
        cswap(d[0], r[0], d[1], r[1]);
        cswap(d[2], r[2], d[3], r[3]);
        cswap(d[0], r[0], d[2], r[2]);
        cswap(d[1], r[1], d[3], r[3]);
        cswap(d[1], r[1], d[2], r[2]);
        int q = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) q += d[c] < best_sq ? 1 : 0;
        if (q > 0) {
          if (st.sp + (q - 1) > Stack::kDepth) return false;
#pragma unroll
          for (int c = 3; c >= 1; --c)
            if (c < q) st.push(r[c], d[c]);
          ref = r[0];
          continue;
        }
      } else {
        const uint32_t f0 = leaf_first(ref), cnt = leaf_count(ref);
        for (uint32_t i = 0; i < cnt; ++i) {
          const TriRec t = T.tri(f0 + i);
          ++ctr.tris;
          const float dsq = tri_dist_sq(t, px, py, pz);
          if (dsq < best_sq) {
            best_sq = dsq;
            best_tri = f0 + i;
          }
        }
      }
    }
    // pop the next candidate that can still beat best_sq
    have = false;
    while (st.sp > 0) {
      const uint2 e = st.pop();
      if (__uint_as_float(e.y) < best_sq) {
        ref = e.x;
        have = true;
        break;
      }
    }
    if (!have) return true;
  }
}

__device__ __forceinline__ void finish_query(const TriRec* __restrict__ tris, uint32_t num_tris, uint32_t best_tri,
                                          float best_sq,
                                             float px, float py, float pz, int64_t qi, const QueryOut& out,
                                             const SignArgs& sg, bool do_sign) {
  float cx = px, cy = py, cz = pz;
  int32_t face = -1;
  float u = 0.f, v = 0.f, w = 0.f;
  float dist = sqrtf(best_sq);
  if (best_tri != 0xffffffffu) {
    const TriRec t = load_tri(tris, best_tri < num_tris ? best_tri : 0u);
    face = __float_as_int(t.a.w);
    const V3<float> a = mk(t.a.x, t.a.y, t.a.z), b = mk(t.b.x, t.b.y, t.b.z), c = mk(t.c.x, t.c.y, t.c.z);
    const V3<float> p = mk(px, py, pz);
    V3<float> cp;
    if (t.c.w < 0.f) {  // near-degenerate
      const V3<double> cd = TriEval<double>::closest(mk<double>(px, py, pz), mk<double>(a.x, a.y, a.z),
                                                     mk<double>(b.x, b.y, b.z), mk<double>(c.x, c.y, c.z));
      cp = mk((float)cd.x, (float)cd.y, (float)cd.z);
    } else {
      cp = TriEval<float>::closest(p, a, b, c);
    }
    cx = cp.x; cy = cp.y; cz = cp.z;
    const V3<float> bc = TriEval<float>::bary(cp, a, b, c);
    u = bc.x; v = bc.y; w = bc.z;
    if (do_sign) {
      // Baerentzen-Aanaes pseudo-normal selected from the barycentrics
      const float eps = 1e-4f;
      const bool z0 = u < eps, z1 = v < eps, z2 = w < eps;
      const int nz = (int)z0 + (int)z1 + (int)z2;
      const float* nrm = sg.face_normals + 3 * (int64_t)face;
      if (sg.edge_pn == nullptr) {
        // face normals only (caller supplied vertex normals)
      } else if (nz == 2) {
        const int dom = !z0 ? 0 : (!z1 ? 1 : 2);
        const int64_t vid = sg.faces[3 * (int64_t)face + dom];
        nrm = sg.vertex_pn + 3 * vid;
      } else if (nz == 1) {
        const int zi = z0 ? 0 : (z1 ? 1 : 2);
        const int he = zi == 0 ? 1 : (zi == 1 ? 2 : 0);
        const int64_t eid = sg.he_edge_idx[3 * (int64_t)face + he];
        nrm = sg.edge_pn + 3 * eid;
      }
      const float nx = __ldg(nrm), ny = __ldg(nrm + 1), nzv = __ldg(nrm + 2);
      float s;
      if (dist < 1e-3f) {
        // near the surface the sign is decided in FP64 from an FP64 closest point
        const V3<double> cd = TriEval<double>::closest(mk<double>(px, py, pz), mk<double>(a.x, a.y, a.z),
                                                       mk<double>(b.x, b.y, b.z), mk<double>(c.x, c.y, c.z));
        const double dd = ((double)px - cd.x) * nx + ((double)py - cd.y) * ny + ((double)pz - cd.z) * nzv;
        s = dd < 0.0 ? -1.f : 1.f;
      } else {
        const float dd = (px - cx) * nx + (py - cy) * ny + (pz - cz) * nzv;
        s = dd < 0.f ? -1.f : 1.f;
      }
      dist *= s;
    }
  }
  out.dist[qi] = dist;
  out.fid[qi] = face;
  out.cp[3 * qi] = cx;
  out.cp[3 * qi + 1] = cy;
  out.cp[3 * qi + 2] = cz;
  if (out.uvw && best_tri != 0xffffffffu) {
    out.uvw[3 * qi] = u;
    out.uvw[3 * qi + 1] = v;
    out.uvw[3 * qi + 2] = w;
  }
}

__device__ __forceinline__ void flush_counters(const Counters& c, unsigned long long* stats) {
  unsigned long long a = warp_reduce_sum(c.nodes), b = warp_reduce_sum(c.tris);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(stats, a);
    atomicAdd(stats + 1, b);
  }
}

// Greedy root-to-leaf probe: follows the nearest child and tests that
// leaf's triangles.  Gives a real triangle (and its distance) that seeds the
// pruning radius of the full traversal.
template <typename Tree>
__device__ __forceinline__ void probe(const Tree& T, float px, float py, float pz, uint32_t& tri, float& dsq,
                                     Counters& ctr, uint32_t root = 0u) {
  uint32_t ref = root;
  while (!ref_is_leaf(ref)) {
    ++ctr.nodes;
    const int4* np = T.node(ref);
    const int4 w0 = __ldg(np), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3);
    const float ox = __int_as_float(w0.x), oy = __int_as_float(w0.y), oz = __int_as_float(w0.z);
    const uint32_t meta = (uint32_t)w0.w;
    const float sx = __uint_as_float((meta & 0xffu) << 23);
    const float sy = __uint_as_float(((meta >> 8) & 0xffu) << 23);
    const float sz = __uint_as_float(((meta >> 16) & 0xffu) << 23);
    const uint32_t r[4] = {(uint32_t)w2.z, (uint32_t)w2.w, (uint32_t)w3.x, (uint32_t)w3.y};
    const int nch = (int)(meta >> 24);
    float bd = INFINITY;
    uint32_t br = r[0];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float lx = dequant((uint32_t)w1.x, c, sx, ox);
      const float ly = dequant((uint32_t)w1.y, c, sy, oy);
      const float lz = dequant((uint32_t)w1.z, c, sz, oz);
      const float hx = dequant((uint32_t)w1.w, c, sx, ox);
      const float hy = dequant((uint32_t)w2.x, c, sy, oy);
      const float hz = dequant((uint32_t)w2.y, c, sz, oz);
      const float d = c < nch ? box_dist_sq(px, py, pz, lx, ly, lz, hx, hy, hz) : INFINITY;
      if (d < bd) { bd = d; br = r[c]; }
    }
    ref = br;
  }
  const uint32_t f0 = leaf_first(ref), cnt = leaf_count(ref);
  dsq = INFINITY;
  tri = f0;
  for (uint32_t i = 0; i < cnt; ++i) {
    ++ctr.tris;
    const float d = tri_dist_sq(T.tri(f0 + i), px, py, pz);
    if (d < dsq) { dsq = d; tri = f0 + i; }
  }
}

// Each thread walks `chunk` consecutive Morton-sorted queries.  The pruning
// radius of a query starts just above its distance to the previous query's
// closest triangle (a greedy probe for the first one), so a valid triangle
// always lies inside it and the traversal returns exactly what an
// unbounded traversal returns: the nodes it skips all lie at or beyond a
// distance some tested triangle already beats or ties earlier in the same
// nearest-first order.  An external bound, when given, tightens the radius
// further; if it excludes every triangle the query is re-run unbounded.
template <bool kStats>
__global__ void __launch_bounds__(kUdfThreads)
    udf_kernel(TreeT<false> T, const float* __restrict__ pts,
               int64_t n, int chunk, const uint32_t* __restrict__ perm, const float* __restrict__ bound,
               Best out, unsigned long long* stats, uint32_t* __restrict__ rerun, uint32_t* __restrict__ nrerun) {
  pdl_wait();
  __shared__ uint2 s_stack[kSharedDepth * kUdfThreads];
  __shared__ uint32_t s_next[kUdfThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // each warp owns 32 * chunk consecutive (sorted) queries and hands them out
  // to its lanes as they finish, so fast lanes do not idle behind slow ones
  const int64_t w0 = ((int64_t)blockIdx.x * (kUdfThreads / 32) + warp) * 32 * chunk;
  const int64_t w1 = w0 + 32 * chunk < n ? w0 + 32 * chunk : n;
  if (lane == 0) s_next[warp] = 32;
  __syncwarp();
  Counters ctr{0, 0};
  uint32_t prev = 0xffffffffu;
  int64_t k = w0 + lane;
  while (k < w1) {
    const int64_t qi = perm ? (int64_t)perm[k] : k;
    const float px = pts[3 * qi], py = pts[3 * qi + 1], pz = pts[3 * qi + 2];
    uint32_t seed_tri;
    float seed_sq;
    if (prev != 0xffffffffu) {
      seed_tri = prev;
      ++ctr.tris;
      seed_sq = tri_dist_sq(T.tri(prev), px, py, pz);
    } else {
      probe(T, px, py, pz, seed_tri, seed_sq, ctr);
    }
    // strictly above the seed distance so the seed triangle itself qualifies
    float best_sq = seed_sq < INFINITY ? nextafterf(seed_sq, INFINITY) : INFINITY;
    if (bound) {
      const float b = bound[qi];
      const float bsq = b * b;
      if (bsq >= 0.f && bsq < best_sq) best_sq = bsq;
    }
    uint32_t best_tri = 0xffffffffu;
    SharedStack st{s_stack + threadIdx.x, 0};
    const bool ok = traverse(T, px, py, pz, st, best_sq, best_tri, ctr);
    if (!ok || best_tri == 0xffffffffu) {
      // stack overflow, or an external bound excluded every triangle
      const uint32_t slot = atomicAdd(nrerun, 1u);
      rerun[slot] = (uint32_t)k;
      prev = 0xffffffffu;
    } else {
      out.tri[qi] = best_tri;
      out.sq[qi] = best_sq;
      prev = best_tri;
    }
    k = w0 + (int64_t)atomicAdd(&s_next[warp], 1u);
  }
  if (kStats) {
    __syncwarp();
    flush_counters(ctr, stats);
  }
}



// Children c0 .. c0 + kC - 1 of a node: box distance d, reference r (0xffffffff
// for no child) and the value e >= d that prunes the child, the larger of the
// box and the disc distance.  The disc is read only for a child whose box
// still qualifies against `best`.  ties: bit x - 1 set when the reference of
// sibling c ^ x is smaller.
template <bool kRecords, int kC, typename Tree>
__device__ __forceinline__ void node_child(const Tree& T, uint32_t ref, int c0, float px, float py, float pz,
                                           float best, float d[kC], uint32_t r[kC], float e[kC], uint32_t ties[kC]) {
  if (kRecords && ref < T.num_children) {
    const BoxRec* rec = T.children.boxes + 4 * (size_t)ref + c0;
    float4 a[kC], b[kC];
#pragma unroll
    for (int j = 0; j < kC; ++j) ldg256(rec + j, a[j], b[j]);
#pragma unroll
    for (int j = 0; j < kC; ++j) {
      r[j] = __float_as_uint(b[j].z);
      ties[j] = __float_as_uint(b[j].w);
      d[j] = r[j] != 0xffffffffu ? box_dist_sq(px, py, pz, a[j].x, a[j].y, a[j].z, a[j].w, b[j].x, b[j].y) : INFINITY;
      e[j] = d[j];
    }
#pragma unroll
    for (int j = 0; j < kC; ++j)
      if (d[j] < best && (ref_is_leaf(r[j]) || r[j] < T.num_children))
        e[j] = fmaxf(d[j], disc_dist_sq(ref_is_leaf(r[j]) ? T.children.leaf_discs + leaf_first(r[j])
                                                          : T.children.node_discs + r[j],
                                        px, py, pz));
    return;
  }
  const WideNode* nd = reinterpret_cast<const WideNode*>(T.node(ref));
  const int4 w0 = __ldg(reinterpret_cast<const int4*>(nd)), w1 = __ldg(reinterpret_cast<const int4*>(nd) + 1);
  const int2 w2 = __ldg(reinterpret_cast<const int2*>(nd) + 4);
  const uint32_t meta = (uint32_t)w0.w;
  const int nch = (int)(meta >> 24);
  const float sx = __uint_as_float((meta & 0xffu) << 23);
  const float sy = __uint_as_float(((meta >> 8) & 0xffu) << 23);
  const float sz = __uint_as_float(((meta >> 16) & 0xffu) << 23);
  const float ox = __int_as_float(w0.x), oy = __int_as_float(w0.y), oz = __int_as_float(w0.z);
#pragma unroll
  for (int j = 0; j < kC; ++j) {
    const int c = c0 + j;
    r[j] = __ldg(nd->ref + c);
    ties[j] = 0;
#pragma unroll
    for (int x = 1; x < 4; ++x) ties[j] |= __ldg(nd->ref + (c ^ x)) < r[j] ? 1u << (x - 1) : 0u;
    const float lx = dequant((uint32_t)w1.x, c, sx, ox);
    const float ly = dequant((uint32_t)w1.y, c, sy, oy);
    const float lz = dequant((uint32_t)w1.z, c, sz, oz);
    const float hx = dequant((uint32_t)w1.w, c, sx, ox);
    const float hy = dequant((uint32_t)w2.x, c, sy, oy);
    const float hz = dequant((uint32_t)w2.y, c, sz, oz);
    d[j] = c < nch ? box_dist_sq(px, py, pz, lx, ly, lz, hx, hy, hz) : INFINITY;
    e[j] = d[j];
  }
}

// ---------------------------------------------------------------------------
// group traversal
// ---------------------------------------------------------------------------
// kG lanes (4 or 2) walk the tree for one query, 32 / kG queries a warp: at a
// node each lane tests 4 / kG children (box, then disc) and the group orders
// and pushes them by shuffles; all lanes of a group hold the query's state,
// so a warp needs few registers and many warps hide the tree's latency.  A
// warp alternates two phases: node steps for the queries at an inner node
// while enough of them are, then one leaf step for those that have reached a
// leaf (or test their seed triangle).  Every query keeps the nearest-first
// order of traverse(), so results and ties are those of a single walk.
constexpr int kGroupWarps = 4;
// stack entries of a query in shared memory, and further ones in the workspace
// where it has room.  The boxes alone prune less, so that stacks go deeper:
// 1,048,576 queries (1,310,720 triangles) without room in the workspace, where a
// query with more entries is run again, took 105 ms at 24 entries, 36.7 at 32
// and 25.6 at 40
template <bool kRecords>
constexpr int kGroupDepth = kRecords ? 24 : 40;
constexpr int kSpillCap = 64;
constexpr int kMaxPool = 64;
constexpr uint32_t kReuseSpan = 64;  // a group's previous result seeds a query this close in the sorted order
// resident blocks an SM (48 registers at 4 lanes, 64 at 2, no spills in the
// loops; one block more at 2 lanes spills and triples the time) and queries at
// a node below which a warp turns to its leaves (16.8M queries, 2 lanes: 37.0,
// 34.9 and 34.1 ms at 6, 8 and 10 of 16; 4 lanes: 38.0, 35.9 and 35.4 ms at 3,
// 4 and 5 of 8)
template <int kG>
constexpr int kGroupBlocks = kG == 4 ? 10 : 8;
template <int kG>
constexpr int kNodeGroups = kG == 4 ? 5 : 10;

template <int kG, bool kRecords>
struct GroupSmem {
  uint2 stack[32 / kG][kGroupDepth<kRecords>];
  uint2 own[32 / kG];                     // a leaf step's queries: first triangle less its first task, first lane
  float trid[32 / kG * kMaxLeafTris];     // distances by task
};

enum : int { kIdle = 0, kSeed = 1, kTrav = 2, kAbandon = 3 };
// radius seeding
enum : uint32_t { kSeedReuse = 1u, kSeedBoundOnly = 2u };

template <int kG, bool kRecords, bool kStats, bool kBatch>
__global__ void __launch_bounds__(kGroupWarps * 32, kGroupBlocks<kG>)
    udf_group_kernel(TreeT<kBatch> T, const float* __restrict__ pts, uint32_t n, const uint32_t* __restrict__ perm,
                     const float* __restrict__ bound, Best out, unsigned long long* stats,
                     uint32_t* __restrict__ rerun, uint32_t* __restrict__ nrerun, uint32_t* __restrict__ pool_counter,
                     uint2* __restrict__ spill, uint32_t spill_owners, uint32_t seeding, MeshSel sel, uint32_t pool,
                     int groups) {
  pdl_wait();
  constexpr int kC = 4 / kG;  // children a lane
  constexpr unsigned lead = kG == 4 ? 0x11111111u : 0x55555555u, gmask = (1u << kG) - 1u;
  constexpr int kDepth = kGroupDepth<kRecords>;
  __shared__ GroupSmem<kG, kRecords> smem[kGroupWarps];
  const int lane = threadIdx.x & 31, c = lane & (kG - 1), base = lane & ~(kG - 1);
  const unsigned FULL = 0xffffffffu;
  GroupSmem<kG, kRecords>& S = smem[threadIdx.x >> 5];
  uint2* stack = S.stack[lane / kG];
  // persistent warps: pools of consecutive (sorted) queries are taken from a
  // global counter; inside a pool, groups take queries as they finish
  uint32_t pos = 0, end = 0;
  bool exhausted = false;
  Counters ctr{0, 0};

  uint32_t k = 0;  // the query's place in the sorted order
  int phase = kIdle;
  uint32_t ref = 0, prev = 0xffffffffu, best_tri = 0xffffffffu, root = 0u, prev_root = 0u;
  float best_sq = INFINITY, px = 0.f, py = 0.f, pz = 0.f, bsq = INFINITY;
  bool have = false;    // ref is the item to process
  bool reused = false;  // the query's radius is seeded by the previous query's triangle
  bool greedy = false;  // descending to the nearest child's leaf for a seed
  int sp = 0;
  unsigned long long rounds = 0;

  // entry i >= kDepth of the query's stack, in the workspace, and the
  // stack's capacity: kDepth, and kSpillCap more where the workspace has
  // room for this group
  auto spill_at = [&](int i) -> uint2* {
    const uint32_t owner = (blockIdx.x * (kGroupWarps * 32) + threadIdx.x) / kG;
    return spill + (size_t)owner * kSpillCap + (i - kDepth);
  };
  auto capacity = [&]() -> int {
    const uint32_t owner = (blockIdx.x * (kGroupWarps * 32) + threadIdx.x) / kG;
    return owner < spill_owners ? kDepth + kSpillCap : kDepth;
  };

  auto start = [&](uint32_t knew) {
    const uint32_t qi = perm ? perm[knew] : knew;
    root = kBatch ? sel.root_of(qi) : 0u;
    px = pts[3 * (int64_t)qi]; py = pts[3 * (int64_t)qi + 1]; pz = pts[3 * (int64_t)qi + 2];
    bsq = INFINITY;
    if (bound) {
      const float b = bound[qi];
      if (b * b >= 0.f) bsq = b * b;
    }
    best_sq = bsq;
    best_tri = 0xffffffffu;
    sp = 0;
    ref = root;
    have = true;
    phase = kTrav;
    // the previous result seeds the radius of a nearby query in the sorted
    // order (a greedy descent when that is not wanted), unless a finite
    // caller bound alone is asked to; a query without a near previous one
    // starts without a radius, which costs less than a descent for one
    const bool alone = (seeding & kSeedBoundOnly) && bsq < INFINITY;
    greedy = !alone && !(seeding & kSeedReuse);
    reused = !alone && (seeding & kSeedReuse) && prev != 0xffffffffu && (!kBatch || root == prev_root) &&
             knew - k <= kReuseSpan;
    if (reused) {
      phase = kSeed;
      have = false;
    }
    k = knew;
    if (kBatch) prev_root = root;
  };

  // hands new queries to the groups in `want` (bits of their first lanes;
  // warp-uniform bookkeeping)
  auto distribute = [&](unsigned want) {
    while (want) {
      if (pos >= end) {
        if (exhausted) break;
        uint32_t p = 0;
        if (lane == 0) p = atomicAdd(pool_counter, 1u);
        p = __shfl_sync(FULL, p, 0);
        const uint64_t first = (uint64_t)p * pool;
        if (first >= n) { exhausted = true; break; }
        pos = (uint32_t)first;
        end = n - pos < pool ? n : pos + pool;
      }
      const uint32_t avail = end - pos, cnt = __popc(want);
      const uint32_t take = avail < cnt ? avail : cnt;
      const uint32_t rank = __popc(want & ((1u << base) - 1u));
      const bool mine = ((want >> base) & 1u) && rank < take;
      if (mine) start(pos + rank);
      pos += take;
      want &= ~__ballot_sync(FULL, mine);
    }
  };

  // pops an item for every group without one: its lanes look at the top kG
  // entries at once
  auto pop = [&]() {
    bool need = phase == kTrav && !have && sp > 0;
    while (__any_sync(FULL, need)) {
      uint2 t = make_uint2(0u, 0x7f800000u);
      const int i = sp - 1 - c;
      if (need && i >= 0) t = i < kDepth ? stack[i] : *spill_at(i);
      const bool good = need && i >= 0 && __uint_as_float(t.y) < best_sq;
      const unsigned gm = (__ballot_sync(FULL, good) >> base) & gmask;
      const int f = __ffs(gm) - 1;
      const uint32_t pr = __shfl_sync(FULL, t.x, base + (f & (kG - 1)));
      if (need) {
        if (gm) {
          ref = pr;
          have = true;
          sp -= f + 1;
        } else {
          sp = sp > kG ? sp - kG : 0;
        }
      }
      need = phase == kTrav && !have && sp > 0;
    }
  };

  distribute(groups >= 32 / kG ? lead : lead & ((1u << (kG * groups)) - 1u));

  while (__any_sync(FULL, phase != kIdle)) {
    if (kStats) ++rounds;
    // (a) node steps
    for (;;) {
      const bool at = phase == kTrav && have && !ref_is_leaf(ref);
      float d[kC], e[kC];
      uint32_t r[kC], ties[kC];
#pragma unroll
      for (int j = 0; j < kC; ++j) {
        d[j] = e[j] = INFINITY;
        r[j] = 0u;
        ties[j] = 0u;
      }
      if (at) {
        if (kStats && c == 0) ++ctr.nodes;
        node_child<kRecords, kC>(T, ref, c * kC, px, py, pz, best_sq, d, r, e, ties);
      }
      // a child is dropped by e (box and disc), visited in order of d (the box
      // alone), so the discs change which children are visited, never their
      // order; rank: the child's place in (distance, ref) order among the
      // qualifying ones, by the distances' bits, which are never negative.  A
      // greedy descent takes any child there is, also where every distance
      // overflows (infinite or huge queries), so it always ends at a leaf
      bool ok[kC];
      int key[kC], rank[kC], q = 0;
      uint32_t next = 0u;
#pragma unroll
      for (int j = 0; j < kC; ++j) {
        ok[j] = e[j] < best_sq || (greedy && r[j] != 0xffffffffu);
        key[j] = ok[j] ? __float_as_int(d[j]) : 0x7f800000;
        q += __popc((__ballot_sync(FULL, ok[j]) >> base) & gmask);
      }
      if (kG == 4) {
        rank[0] = 0;
#pragma unroll
        for (int x = 1; x < 4; ++x)
          rank[0] += __shfl_xor_sync(FULL, key[0], x) < key[0] + (int)((ties[0] >> (x - 1)) & 1u) ? 1 : 0;
      } else {
        const int o0 = __shfl_xor_sync(FULL, key[0], 1), o1 = __shfl_xor_sync(FULL, key[kC - 1], 1);
        const uint32_t t0 = ties[0], t1 = ties[kC - 1];
        const int k0 = key[0], k1 = key[kC - 1];
        rank[0] = (k1 < k0 + (int)(t0 & 1u)) + (o0 < k0 + (int)((t0 >> 1) & 1u)) + (o1 < k0 + (int)(t0 >> 2));
        rank[kC - 1] = (k0 < k1 + (int)(t1 & 1u)) + (o1 < k1 + (int)((t1 >> 1) & 1u)) + (o0 < k1 + (int)(t1 >> 2));
      }
#pragma unroll
      for (int j = 0; j < kC; ++j) next |= ok[j] && rank[j] == 0 ? r[j] : 0u;
#pragma unroll
      for (int x = 1; x < kG; x <<= 1) next |= __shfl_xor_sync(FULL, next, x);
      if (at) {
        if (greedy) {
          ref = next;
        } else if (q > 0) {
          if (sp + q - 1 > kDepth && sp + q - 1 > capacity()) {
            // no room: the deep-stack kernel re-runs the query
            phase = kAbandon;
            have = false;
          } else {
#pragma unroll
            for (int j = 0; j < kC; ++j) {
              const int i = sp + q - 1 - rank[j];
              if (ok[j] && rank[j] > 0) {
                if (i < kDepth) stack[i] = make_uint2(r[j], __float_as_uint(e[j]));
                else *spill_at(i) = make_uint2(r[j], __float_as_uint(e[j]));
              }
            }
            sp += q - 1;
            ref = next;
          }
        } else {
          have = false;
        }
      }
      __syncwarp();
      pop();
      const unsigned at_node = __ballot_sync(FULL, phase == kTrav && have && !ref_is_leaf(ref));
      if (__popc(at_node) >= kG * kNodeGroups<kG>) continue;
      if (at_node == 0) break;
      // few queries at nodes: go on only if none waits for a leaf step or its end
      if (__any_sync(FULL, phase == kSeed || phase == kAbandon || (phase == kTrav && (!have || ref_is_leaf(ref)))))
        break;
    }
    // (b) leaf step
    uint32_t cnt = phase == kSeed ? 1u : (phase == kTrav && have && ref_is_leaf(ref) ? leaf_count(ref) : 0u);
    if (__any_sync(FULL, cnt > 0u)) {
      if (kStats && c == 0) ctr.tris += cnt;
      float dmin = INFINITY;
      uint32_t imin = 0xffffffffu;
      if (kG == 4) {
        // every fourth triangle a lane
        for (uint32_t i = c; i < cnt; i += 4) {
          const uint32_t ti = (phase == kSeed ? prev : leaf_first(ref)) + i;
          const TriRec tr = T.tri(ti);
          float dd;
          if (tr.c.w < 0.f) {
            // near-degenerate: the FP64 evaluation is a call, and what stays
            // live across a call is spilled in the hot loops as well; so the
            // state is put aside by hand here and dead until it is read back
            volatile uint32_t keep[20];
            keep[0] = k; keep[1] = (uint32_t)phase; keep[2] = ref; keep[3] = prev; keep[4] = best_tri;
            keep[5] = root; keep[6] = prev_root; keep[7] = __float_as_uint(best_sq); keep[8] = __float_as_uint(px);
            keep[9] = __float_as_uint(py); keep[10] = __float_as_uint(pz); keep[11] = __float_as_uint(bsq);
            keep[12] = (uint32_t)sp; keep[13] = pos; keep[14] = end; keep[15] = i;
            keep[16] = __float_as_uint(dmin); keep[17] = imin; keep[18] = cnt;
            keep[19] = (have ? 1u : 0u) | (reused ? 2u : 0u) | (exhausted ? 4u : 0u) | (greedy ? 8u : 0u);
            dd = tri_dist_sq_f64(tr.a.x, tr.a.y, tr.a.z, tr.b.x, tr.b.y, tr.b.z, tr.c.x, tr.c.y, tr.c.z, px, py, pz);
            k = keep[0]; phase = (int)keep[1]; ref = keep[2]; prev = keep[3]; best_tri = keep[4];
            root = keep[5]; prev_root = keep[6]; best_sq = __uint_as_float(keep[7]); px = __uint_as_float(keep[8]);
            py = __uint_as_float(keep[9]); pz = __uint_as_float(keep[10]); bsq = __uint_as_float(keep[11]);
            sp = (int)keep[12]; pos = keep[13]; end = keep[14]; i = keep[15];
            dmin = __uint_as_float(keep[16]); imin = keep[17]; cnt = keep[18];
            const uint32_t fl = keep[19];
            have = (fl & 1u) != 0u; reused = (fl & 2u) != 0u; exhausted = (fl & 4u) != 0u; greedy = (fl & 8u) != 0u;
          } else {
            dd = dist_sq_bary(mk(px, py, pz), mk(tr.a.x, tr.a.y, tr.a.z), mk(tr.b.x, tr.b.y, tr.b.z),
                              mk(tr.c.x, tr.c.y, tr.c.z), tr.c.w, tr.b.w, tr.r.w, tr.r.x, tr.r.y, tr.r.z);
          }
          if (dd < dmin) { dmin = dd; imin = (phase == kSeed ? prev : leaf_first(ref)) + i; }
        }
      } else {
        // the triangles of all waiting queries as one list of tasks, a lane each
        uint32_t off = cnt;  // tasks up to and with this query's
#pragma unroll
        for (int o = kG; o < 32; o <<= 1) {
          const uint32_t v = __shfl_up_sync(FULL, off, o);
          if (lane >= o) off += v;
        }
        uint32_t total = __shfl_sync(FULL, off, 31);
        off -= cnt;
        const unsigned owners = __ballot_sync(FULL, cnt > 0u) & lead;
        if (c == 0 && cnt > 0u)
          S.own[__popc(owners & ((1u << base) - 1u))] =
              make_uint2((phase == kSeed ? prev : leaf_first(ref)) - off, (uint32_t)lane);
        __syncwarp();
        int before = -1;  // owners whose first task lies before this group of 32
        for (uint32_t t0 = 0; t0 < total; t0 += 32) {
          const unsigned firsts =
              __reduce_or_sync(FULL, cnt > 0u && (off >> 5) == (t0 >> 5) ? 1u << (off & 31u) : 0u);
          const uint2 w = S.own[before + __popc(firsts & (0xffffffffu >> (31 - lane)))];
          before += __popc(firsts);
          const float qx = __shfl_sync(FULL, px, w.y), qy = __shfl_sync(FULL, py, w.y),
                      qz = __shfl_sync(FULL, pz, w.y);
          const uint32_t t = t0 + (uint32_t)lane;
          if (t < total) {
            const TriRec tr = T.tri(w.x + t);
            if (tr.c.w < 0.f) {
              // as above
              volatile uint32_t keep[21];
              keep[0] = k; keep[1] = (uint32_t)phase; keep[2] = ref; keep[3] = prev; keep[4] = best_tri;
              keep[5] = root; keep[6] = prev_root; keep[7] = __float_as_uint(best_sq); keep[8] = __float_as_uint(px);
              keep[9] = __float_as_uint(py); keep[10] = __float_as_uint(pz); keep[11] = __float_as_uint(bsq);
              keep[12] = (uint32_t)sp; keep[13] = pos; keep[14] = end; keep[15] = t0;
              keep[16] = off; keep[17] = total; keep[18] = (uint32_t)before; keep[19] = cnt;
              keep[20] = (have ? 1u : 0u) | (reused ? 2u : 0u) | (exhausted ? 4u : 0u) | (greedy ? 8u : 0u);
              S.trid[t0 + lane] = tri_dist_sq_f64(tr.a.x, tr.a.y, tr.a.z, tr.b.x, tr.b.y, tr.b.z, tr.c.x, tr.c.y,
                                                  tr.c.z, qx, qy, qz);
              k = keep[0]; phase = (int)keep[1]; ref = keep[2]; prev = keep[3]; best_tri = keep[4];
              root = keep[5]; prev_root = keep[6]; best_sq = __uint_as_float(keep[7]); px = __uint_as_float(keep[8]);
              py = __uint_as_float(keep[9]); pz = __uint_as_float(keep[10]); bsq = __uint_as_float(keep[11]);
              sp = (int)keep[12]; pos = keep[13]; end = keep[14]; t0 = keep[15];
              off = keep[16]; total = keep[17]; before = (int)keep[18]; cnt = keep[19];
              const uint32_t fl = keep[20];
              have = (fl & 1u) != 0u; reused = (fl & 2u) != 0u; exhausted = (fl & 4u) != 0u; greedy = (fl & 8u) != 0u;
            } else {
              S.trid[t] = dist_sq_bary(mk(qx, qy, qz), mk(tr.a.x, tr.a.y, tr.a.z), mk(tr.b.x, tr.b.y, tr.b.z),
                                       mk(tr.c.x, tr.c.y, tr.c.z), tr.c.w, tr.b.w, tr.r.w, tr.r.x, tr.r.y, tr.r.z);
            }
          }
        }
        __syncwarp();
        const uint32_t f0 = phase == kSeed ? prev : leaf_first(ref);
        for (uint32_t i = c; i < cnt; i += kG) {
          const float dd = S.trid[off + i];
          if (dd < dmin) { dmin = dd; imin = f0 + i; }
        }
      }
      // the first of the smallest, as one lane testing them in order finds it
#pragma unroll
      for (int x = 1; x < kG; x <<= 1) {
        const float od = __shfl_xor_sync(FULL, dmin, x);
        const uint32_t oi = __shfl_xor_sync(FULL, imin, x);
        if (child_less(od, oi, dmin, imin)) { dmin = od; imin = oi; }
      }
      if (cnt > 0u) {
        if (phase == kTrav && !greedy) {
          if (dmin < best_sq) {
            best_sq = dmin;
            best_tri = imin;
          }
          have = false;
        } else {
          // radius just above the seed triangle's distance
          float b = dmin < INFINITY ? nextafterf(dmin, INFINITY) : INFINITY;
          if (bsq < b) b = bsq;
          best_sq = b;
          reused = true;
          greedy = false;
          phase = kTrav;
          ref = root;
          have = true;
        }
      }
      __syncwarp();
    }
    pop();
    // (c) finished queries emit, their groups take new ones
    bool done = phase == kTrav && !have;
    if (done && best_tri == 0xffffffffu && (bsq < INFINITY || reused)) {
      // the caller's bound excluded every triangle, or the seed triangle's own
      // box rounds to beyond it (flat axis-aligned faces): run the query again
      // in place, without the bound, then without the seed
      const bool again = reused && bsq < INFINITY && prev != 0xffffffffu && (seeding & kSeedReuse);
      bsq = INFINITY;
      best_sq = INFINITY;
      reused = again;
      sp = 0;
      ref = root;
      have = !again;
      phase = again ? kSeed : kTrav;
      done = false;
    }
    if (phase == kAbandon) done = true;
    const unsigned dmask = __ballot_sync(FULL, done);
    if (dmask) {
      if (done) {
        if (phase != kAbandon && best_tri != 0xffffffffu) {
          if (c == 0) {
            const uint32_t at = perm ? perm[k] : k;
            out.tri[at] = best_tri;
            out.sq[at] = best_sq;
          }
          prev = best_tri;
        } else {
          if (c == 0) rerun[atomicAdd(nrerun, 1u)] = k;
          prev = 0xffffffffu;
        }
        phase = kIdle;
      }
      distribute(dmask & lead);
    }
  }
  if (kStats) {
    flush_counters(ctr, stats);
    if (lane == 0) atomicAdd(stats + 3, rounds);
  }
}


template <bool kStats, bool kBatch>
__global__ void __launch_bounds__(64)
    udf_rerun_kernel(TreeT<kBatch> T, const float* __restrict__ pts, const uint32_t* __restrict__ perm,
                     const uint32_t* __restrict__ rerun, const uint32_t* __restrict__ nrerun, Best out,
                     unsigned long long* stats, uint32_t* __restrict__ overflow, uint32_t* __restrict__ total_reruns,
                     MeshSel sel) {
  pdl_wait();
  const uint32_t m = *nrerun;
  if (blockIdx.x == 0 && threadIdx.x == 0 && m > 0) atomicAdd(total_reruns, m);
  Counters ctr{0, 0};
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t k = rerun[t];
    const int64_t qi = perm ? perm[k] : k;
    const float px = pts[3 * qi], py = pts[3 * qi + 1], pz = pts[3 * qi + 2];
    uint32_t seed_tri;
    float seed_sq;
    const uint32_t root = kBatch ? sel.root_of(qi) : 0u;
    probe(T, px, py, pz, seed_tri, seed_sq, ctr, root);
    float best_sq = seed_sq < INFINITY ? nextafterf(seed_sq, INFINITY) : INFINITY;
    uint32_t best_tri = 0xffffffffu;
    LocalStack st;
    st.sp = 0;
    bool ok = traverse(T, px, py, pz, st, best_sq, best_tri, ctr, root);
    if (ok && best_tri == 0xffffffffu) {
      // the probed triangle's own box rounds to beyond it: no radius
      best_sq = INFINITY;
      st.sp = 0;
      ok = traverse(T, px, py, pz, st, best_sq, best_tri, ctr, root);
    }
    if (!ok) atomicExch(overflow, 1u);
    out.tri[qi] = best_tri;
    out.sq[qi] = best_sq;
  }
  if (kStats && (ctr.nodes | ctr.tris)) {
    atomicAdd(stats, ctr.nodes);
    atomicAdd(stats + 1, ctr.tris);
  }
}

// The caller's outputs from the traversal's results, one thread per query in the
// caller's order: points, results and outputs are read and written in order, and
// only the triangle records, which L2 holds, are gathered.  (In sorted order,
// with points and outputs scattered, 16.8M queries took 3.29 ms.)  A kernel of
// its own because the closest point, barycentrics and sign would cost the
// traversal its registers
// (in it: 192 B of spills a lane, which with 24 warps an SM overflow L1).
template <bool kSign>
__global__ void __launch_bounds__(256)
    udf_finish_kernel(const TriRec* __restrict__ tris, uint32_t num_tris, const float* __restrict__ pts, int64_t n,
                      Best best, QueryOut out, SignArgs sg) {
  pdl_wait();
  const int64_t qi = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (qi >= n) return;
  finish_query(tris, num_tris, best.tri[qi], best.sq[qi], pts[3 * qi], pts[3 * qi + 1], pts[3 * qi + 2], qi, out, sg,
               kSign);
}

__global__ void query_morton_kernel(const float* __restrict__ pts, int64_t n, float lox, float loy, float loz,
                                    float inv, float qmax, uint32_t* __restrict__ keys,
                                    uint32_t* __restrict__ vals) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float q[3] = {(pts[3 * i] - lox) * inv, (pts[3 * i + 1] - loy) * inv, (pts[3 * i + 2] - loz) * inv};
  uint32_t code = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float t = fminf(fmaxf(q[a], 0.f), qmax);
    if (!(t == t)) t = 0.f;
    code |= (uint32_t)spread3_21((uint64_t)t) << a;
  }
  keys[i] = code;
  vals[i] = (uint32_t)i;
}

constexpr int kStatusWords = 8;

// Queries are Morton-sorted from kSortMin on, those without child records from
// kSortMinBoxes on.  Below it what the sorted order saves (L1 misses, a seed from
// the neighbour) does not pay for the sort, even for queries in random order.  ms,
// unsorted / sorted, with records:
//                                       300k         700k         1M           1.3M
//   1,310,720 triangles, uniform      1.64 / 1.68  3.47 / 3.32  4.82 / 4.46  6.16 / 5.62
//   the same, half of them near it     1.20 / 1.32  2.45 / 2.53  3.31 / 3.43  4.22 / 4.18
//   20,480 rough triangles, uniform   0.70 / 0.68  1.49 / 1.38  2.08 / 1.92  2.68 / 2.44
//   1,000,000 scattered triangles     0.51 / 0.51  1.18 / 1.07  1.69 / 1.47  2.20 / 1.87
// (the last at 1M, sorted, without records and discs: 1.62) and by boxes alone
// (the first mesh, two lanes, 1M) 26.0 / 30.4 and 14.7 / 19.1.  Below kSortFine 8
// bits an axis (three passes) order as well as 10 (four), above 10 gain about 1%.
constexpr int64_t kSortMin = 7 << 17, kSortMinBoxes = 3 << 19;
inline bool sorted_queries(bool records, int64_t n) { return n >= (records ? kSortMin : kSortMinBoxes); }
constexpr int64_t kSortFine = 8 << 20;

struct UdfWs {
  uint32_t* keys;
  uint32_t* keys_alt;
  uint32_t* vals;
  uint32_t* vals_alt;
  uint32_t* rs_scratch;
  uint32_t* rerun;
  uint32_t* nrerun;  // status words: [0] re-run list length, [1] deep-stack overflow, [2] pool counter,
                     // [3] guard faults, [4] queries re-run in total
  Best best;         // the traversal's results; with a query sort in its key buffers, free after it
  uint2* spill;      // optional overflow stacks (trailing workspace)
  int64_t spill_owners;
};

size_t carve_udf(UdfWs& w, Workspace& ws, int64_t n, uint32_t flags) {
  // status words at the start of the workspace (read by a3d_udf_status)
  w.nrerun = ws.take<uint32_t>(kStatusWords);
  if (flags & A3D_UDF_SORT_QUERIES) {
    w.keys = ws.take<uint32_t>(n);
    w.keys_alt = ws.take<uint32_t>(n);
    w.vals = ws.take<uint32_t>(n);
    w.vals_alt = ws.take<uint32_t>(n);
    w.rs_scratch = ws.take<uint32_t>((int64_t)radix_sort_scratch_elems(n));
    w.best = Best{w.keys, reinterpret_cast<float*>(w.keys_alt)};
  } else {
    w.keys = w.keys_alt = w.vals = w.vals_alt = w.rs_scratch = nullptr;
    w.best.tri = ws.take<uint32_t>(n);
    w.best.sq = ws.take<float>(n);
  }
  w.rerun = ws.take<uint32_t>(n);
  return ws.used;
}

// queries in flight (four lanes each) that get an overflow stack when the
// workspace has room for it (bounded: 148 SMs x 64 warps)
int64_t spill_owner_bound(int64_t n) {
  const int64_t cap = (int64_t)148 * 32 * 16;
  return (n + kGroupWarps) * 16 < cap ? (n + kGroupWarps) * 16 : cap;  // a warp may take one query only
}

// launch shape of the persistent traversal: queries per pool, resident
// blocks per SM (0 = as many as fit)
struct TaskShape {
  int pool;
  int blocks_per_sm;
};

template <int kG, bool kRecords, bool kStats, bool kBatch>
int group_blocks_per_sm(int* out) {
  // per device: a process may drive GPUs of different kinds
  static int cached[kMaxDevices] = {0};
  int dev = 0;
  A3D_CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 0 && dev < kMaxDevices && cached[dev] > 0) {
    *out = cached[dev];
    return A3D_OK;
  }
  int b = 0;
  A3D_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, udf_group_kernel<kG, kRecords, kStats, kBatch>,
                                                             kGroupWarps * 32, 0));
  b = b < 1 ? 1 : b;
  if (dev >= 0 && dev < kMaxDevices) cached[dev] = b;
  *out = b;
  return A3D_OK;
}

template <int kG, bool kRecords, bool kStats, bool kBatch>
int launch_groups(const TreeT<kBatch>& T, const float* pts, int64_t n, const uint32_t* perm, const float* bound,
                  unsigned long long* stats, UdfWs& w, uint32_t seeding, const MeshSel& sel, TaskShape shape,
                  cudaStream_t s) {
  int bps = 0;
  A3D_TRY((group_blocks_per_sm<kG, kRecords, kStats, kBatch>(&bps)));
  if (shape.blocks_per_sm > 0 && shape.blocks_per_sm < bps) bps = shape.blocks_per_sm;
  const int64_t warps = (int64_t)num_sms() * bps * kGroupWarps;
  // few queries: as few a warp as the resident warps allow
  const int64_t per_warp = ceil_div(n, warps);
  const int groups = per_warp < 32 / kG ? (int)per_warp : 32 / kG;
  int64_t pool = shape.pool;
  if (pool <= 0) {
    pool = per_warp / 4;
    pool = pool < groups ? groups : (pool > kMaxPool ? kMaxPool : pool);
  }
  const int64_t want_blocks = ceil_div(ceil_div(n, pool), kGroupWarps);
  const int64_t grid = want_blocks < warps / kGroupWarps ? want_blocks : warps / kGroupWarps;
  const int64_t owners = w.spill == nullptr ? 0 : (w.spill_owners < 0x7fffffff ? w.spill_owners : 0x7fffffff);
  A3D_PDL((udf_group_kernel<kG, kRecords, kStats, kBatch>), dim3((unsigned)grid), dim3(kGroupWarps * 32), 0, s, T, pts,
          (uint32_t)n, perm, bound, w.best, stats, w.rerun, w.nrerun, w.nrerun + 2, w.spill, (uint32_t)owners, seeding,
          sel, (uint32_t)pool, groups);
  return A3D_OK;
}

// From this many queries on two lanes a query, below it four: four take fewer
// steps a query, which counts while the queries in flight do not fill the
// chip, two execute less per query (16.8M queries: 34.1 against 36.6 ms; 24
// meshes with 8.7M: 23.8 against 25.0 with their build; 300k: 0.86 against
// 0.83; 100k: 0.44 against 0.38).
constexpr int64_t kPairMin = 2 << 20;
// The same for the boxes alone, where a query tests ten times the triangles, which
// two lanes a query spread over the warp: 300k / 1M / 4M queries 10.4 / 27.5 / 103
// ms at four lanes, 10.4 / 25.3 / 81 at two against 1,310,720 triangles, 0.94 /
// 2.84 / 9.10 and 0.92 / 2.53 / 8.00 against 20,480.
constexpr int64_t kPairMinBoxes = 3 << 18;

inline bool two_lanes(bool records, int64_t n) { return n >= (records ? kPairMin : kPairMinBoxes); }

// n queries with the kernel of a call of `like` (n itself, but for the
// autotuner's samples)
template <bool kSign, bool kStats, bool kBatch>
int launch_udf(const TreeT<kBatch>& T, const float* pts, int64_t n, int64_t like, const uint32_t* perm, bool coherent,
               const float* bound, const QueryOut& out, const SignArgs& sg, unsigned long long* stats, UdfWs& w,
               uint32_t seeding, const MeshSel& sel, TaskShape shape, cudaStream_t s) {
  if (coherent) {
    const bool records = T.num_children > 0u, two = two_lanes(records, like);
    A3D_TRY(
        records && two ? (launch_groups<2, true, kStats, kBatch>(T, pts, n, perm, bound, stats, w, seeding, sel, shape, s))
        : records ? (launch_groups<4, true, kStats, kBatch>(T, pts, n, perm, bound, stats, w, seeding, sel, shape, s))
        : two ? (launch_groups<2, false, kStats, kBatch>(T, pts, n, perm, bound, stats, w, seeding, sel, shape, s))
              : (launch_groups<4, false, kStats, kBatch>(T, pts, n, perm, bound, stats, w, seeding, sel, shape, s)));
  } else {
    if constexpr (!kBatch) {
      A3D_PDL((udf_kernel<kStats>), dim3((unsigned)ceil_div(n, kUdfThreads)), dim3(kUdfThreads), 0, s, T, pts, n, 1,
              perm, bound, w.best, stats, w.rerun, w.nrerun);
    } else {
      A3D_REQUIRE(false, A3D_ERR_ARGUMENT, "udf: batches are always sorted");
    }
  }
  A3D_LAUNCH_CHECK();
  // the re-run list length is only known on the device (and nearly always 0)
  const int64_t rr_threads = (int64_t)num_sms() * 256;
  A3D_PDL((udf_rerun_kernel<kStats, kBatch>), dim3((unsigned)ceil_div(rr_threads, 64)), dim3(64), 0, s, T, pts, perm,
          w.rerun, w.nrerun, w.best, stats, w.nrerun + 1, w.nrerun + 4, sel);
  A3D_PDL(udf_finish_kernel<kSign>, dim3((unsigned)ceil_div(n, 256)), dim3(256), 0, s, T.tris, T.num_tris, pts, n, w.best,
          out, sg);
  return A3D_OK;
}

// ---------------------------------------------------------------------------
// adjoints
// ---------------------------------------------------------------------------
__global__ void udf_backward_kernel(const float* __restrict__ pts, int64_t n, const float* __restrict__ cp,
                                    const int32_t* __restrict__ fid, const float* __restrict__ uvw,
                                    const float* __restrict__ gd, const int32_t* __restrict__ faces,
                                    float* __restrict__ gp, float* __restrict__ gv) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float dx = pts[3 * i] - cp[3 * i], dy = pts[3 * i + 1] - cp[3 * i + 1], dz = pts[3 * i + 2] - cp[3 * i + 2];
  const float d = sqrtf(dx * dx + dy * dy + dz * dz);
  const float g = gd[i];
  // d|p-c|/dp = (p-c)/|p-c| (zero at the surface, like norm's subgradient)
  const float inv = d > 0.f ? g / d : 0.f;
  const float gx = dx * inv, gy = dy * inv, gz = dz * inv;
  if (gp) {
    gp[3 * i] = gx;
    gp[3 * i + 1] = gy;
    gp[3 * i + 2] = gz;
  }
  const int32_t f = fid[i];
  if (gv && f >= 0 && uvw) {
    // closest-point barycentrics clamped to the simplex (they are exact
    // for the closest point up to rounding)
    float w0 = fmaxf(uvw[3 * i], 0.f), w1 = fmaxf(uvw[3 * i + 1], 0.f), w2 = fmaxf(uvw[3 * i + 2], 0.f);
    const float sw = w0 + w1 + w2;
    if (sw > 0.f) { w0 /= sw; w1 /= sw; w2 /= sw; }
    const float ws[3] = {w0, w1, w2};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int64_t v = faces[3 * (int64_t)f + k];
      atomicAdd(&gv[3 * v], -ws[k] * gx);
      atomicAdd(&gv[3 * v + 1], -ws[k] * gy);
      atomicAdd(&gv[3 * v + 2], -ws[k] * gz);
    }
  }
}

}  // namespace

}  // namespace a3d

using namespace a3d;

namespace a3d {
// Workspace a3d_udf needs at least (without the optional overflow stacks).
size_t udf_required_workspace_bytes(int64_t num_points, uint32_t flags) {
  Workspace ws(nullptr, 0);
  UdfWs w;
  return carve_udf(w, ws, num_points > 0 ? num_points : 1, flags) + 256;
}
}  // namespace a3d

extern "C" size_t a3d_udf_workspace_bytes(int64_t num_points, uint32_t flags) {
  Workspace ws(nullptr, 0);
  UdfWs w;
  const int64_t n = num_points > 0 ? num_points : 1;
  const size_t base = carve_udf(w, ws, n, flags);
  return base + (size_t)spill_owner_bound(n) * kSpillCap * sizeof(uint2) + 512;
}

extern "C" int a3d_udf(const a3d_bvh_view* bvh, const float* points, int64_t num_points, float* distances,
                       int32_t* face_ids, float* closest_points, float* uvw, const a3d_sign_data* sign,
                       const float* bound, unsigned long long* stats, uint32_t flags, void* workspace,
                       size_t workspace_bytes, a3d_stream_t stream) {
  return a3d_udf_children(bvh, nullptr, points, num_points, distances, face_ids, closest_points, uvw, sign, bound,
                          stats, flags, workspace, workspace_bytes, stream);
}

extern "C" int a3d_udf_children(const a3d_bvh_view* bvh, const void* children, const float* points, int64_t num_points,
                             float* distances, int32_t* face_ids, float* closest_points, float* uvw,
                             const a3d_sign_data* sign, const float* bound, unsigned long long* stats, uint32_t flags,
                             void* workspace, size_t workspace_bytes, a3d_stream_t stream_) {
  cudaStream_t s = (cudaStream_t)stream_;
  A3D_REQUIRE(bvh && bvh->nodes && bvh->tris && bvh->num_nodes > 0, A3D_ERR_ARGUMENT, "udf: invalid bvh");
  A3D_REQUIRE(num_points >= 0 && num_points < (1ll << 32), A3D_ERR_ARGUMENT, "udf: bad number of points");
  if (num_points == 0) return A3D_OK;
  A3D_REQUIRE(points && distances && face_ids && closest_points, A3D_ERR_ARGUMENT, "udf: null output");
  A3D_REQUIRE(((uintptr_t)children & 31) == 0, A3D_ERR_ARGUMENT, "udf: child records must be 32-B aligned");
  if (sign) {
    A3D_REQUIRE(sign->face_normals && sign->faces, A3D_ERR_ARGUMENT, "udf: sign data needs face normals and faces");
    const bool all = sign->vertex_pn && sign->edge_pn && sign->he_edge_idx;
    const bool none = !sign->vertex_pn && !sign->edge_pn && !sign->he_edge_idx;
    A3D_REQUIRE(all || none, A3D_ERR_ARGUMENT, "udf: pseudo-normal data must be all present or all absent");
  }
  Workspace ws(workspace, workspace_bytes);
  UdfWs w;
  carve_udf(w, ws, num_points, flags);
  A3D_REQUIRE(workspace && ws.ok(), A3D_ERR_WORKSPACE, "udf: workspace too small");
  // whatever trails the required part holds per-owner overflow stacks
  {
    const uintptr_t base = ((uintptr_t)workspace + ws.used + 255) & ~(uintptr_t)255;
    const uintptr_t endp = (uintptr_t)workspace + workspace_bytes;
    const int64_t owners = base < endp ? (int64_t)((endp - base) / (kSpillCap * sizeof(uint2))) : 0;
    w.spill = owners > 0 ? (uint2*)base : nullptr;
    w.spill_owners = owners;
  }
  const int64_t n = num_points;
  const uint32_t* perm = nullptr;
  const bool sort = (flags & A3D_UDF_SORT_QUERIES) != 0 && sorted_queries(children != nullptr, n);
  if (sort) {
    const float ext[3] = {bvh->hi[0] - bvh->lo[0], bvh->hi[1] - bvh->lo[1], bvh->hi[2] - bvh->lo[2]};
    float emax = fmaxf(ext[0], fmaxf(ext[1], ext[2]));
    emax = emax > 0.f ? emax : 1.f;
    // queries may lie outside the mesh box: use a cube of twice its extent
    const float lo[3] = {0.5f * (bvh->lo[0] + bvh->hi[0]) - emax, 0.5f * (bvh->lo[1] + bvh->hi[1]) - emax,
                         0.5f * (bvh->lo[2] + bvh->hi[2]) - emax};
    const int bits = n < kSortFine ? 8 : 10;
    const float qmax = (float)((1 << bits) - 1);
    A3D_PDL(query_morton_kernel, dim3((unsigned)ceil_div(n, 256)), dim3(256), 0, s, points, n, lo[0], lo[1], lo[2],
            qmax / (2.0f * emax), qmax, w.keys, w.vals);
    bool alt = false;
    A3D_TRY(radix_sort_pairs<uint32_t>(w.keys, w.vals, w.keys_alt, w.vals_alt, n, 0, 3 * bits, w.rs_scratch, &alt, s));
    perm = alt ? w.vals_alt : w.vals;
  }
  // in the caller's order when there are few: the same traversal, no sort
  const bool coherent = (flags & A3D_UDF_SORT_QUERIES) != 0 || (flags & A3D_UDF_ASSUME_SORTED) != 0;
  const uint32_t seeding = ((flags & A3D_UDF_NO_REUSE) ? 0u : kSeedReuse) |
                           ((flags & A3D_UDF_BOUND_SEEDS) && bound ? kSeedBoundOnly : 0u);
  A3D_CUDA_TRY(cudaMemsetAsync(w.nrerun, 0, kStatusWords * sizeof(uint32_t), s));
  const TreeT<false> T{(const WideNode*)bvh->nodes, (const TriRec*)bvh->tris, (uint32_t)bvh->num_nodes,
                       (uint32_t)bvh->num_tris, w.nrerun + 3, ChildRecs(children, bvh->num_nodes),
                       children != nullptr ? (uint32_t)bvh->num_nodes : 0u};
  const MeshSel sel{nullptr, nullptr, 1, 0};
  const TaskShape shape{0, 0};
  QueryOut out{distances, face_ids, closest_points, uvw};
  SignArgs sg{nullptr, nullptr, nullptr, nullptr, nullptr};
  if (sign) {
    const bool pn = sign->edge_pn != nullptr;
    sg = SignArgs{sign->face_normals, pn ? sign->vertex_pn : nullptr, pn ? sign->edge_pn : nullptr,
                  pn ? sign->he_edge_idx : nullptr, sign->faces};
  }
  if (sign) {
    if (stats)
      A3D_TRY((launch_udf<true, true, false>(T, points, n, n, perm, coherent, bound, out, sg, stats, w, seeding, sel,
                                             shape, s)));
    else
      A3D_TRY((launch_udf<true, false, false>(T, points, n, n, perm, coherent, bound, out, sg, stats, w, seeding, sel,
                                              shape, s)));
  } else {
    if (stats)
      A3D_TRY((launch_udf<false, true, false>(T, points, n, n, perm, coherent, bound, out, sg, stats, w, seeding, sel,
                                              shape, s)));
    else
      A3D_TRY((launch_udf<false, false, false>(T, points, n, n, perm, coherent, bound, out, sg, stats, w, seeding, sel,
                                               shape, s)));
  }
  if (stats) {
    // reruns are reported as bound misses / spills (same counter: re-run queries)
    A3D_CUDA_TRY(cudaMemcpyAsync(stats + 2, w.nrerun + 4, sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
  }
  return A3D_OK;
}

extern "C" int a3d_udf_backward(const float* points, int64_t num_points, const float* closest_points,
                                const int32_t* face_ids, const float* uvw, const float* grad_dist,
                                const int32_t* faces, float* grad_points, float* grad_vertices,
                                a3d_stream_t stream_) {
  cudaStream_t s = (cudaStream_t)stream_;
  A3D_REQUIRE(num_points >= 0, A3D_ERR_ARGUMENT, "udf_backward: bad size");
  if (num_points == 0) return A3D_OK;
  A3D_REQUIRE(points && closest_points && grad_dist, A3D_ERR_ARGUMENT, "udf_backward: null input");
  A3D_REQUIRE(!grad_vertices || (face_ids && uvw && faces), A3D_ERR_ARGUMENT,
              "udf_backward: vertex adjoint needs face ids, uvw and faces");
  A3D_PDL(udf_backward_kernel, dim3((unsigned)ceil_div(num_points, 256)), dim3(256), 0, s, points, num_points,
          closest_points, face_ids, uvw, grad_dist, faces, grad_points, grad_vertices);
  return A3D_OK;
}

// ---------------------------------------------------------------------------
// batches of meshes: one sort and one persistent traversal per chunk of
// queries, all meshes together
// ---------------------------------------------------------------------------
namespace a3d {
namespace {

// blocks an SM of a tuning that takes all that fit, whatever the kernel (32: an
// SM's most), so that calls of another size are not held to one kernel's count
constexpr int kAllBlocks = 32;
// queries per traversal launch of a batch (bounds the scratch: ~380 MB)
constexpr int64_t kBatchChunk = 1ll << 24;

__device__ __forceinline__ int segment_of64(const int64_t* __restrict__ off, int nseg, int64_t i) {
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= i) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// key = mesh id above the Morton code of the query in a cube of twice its
// mesh's extent about the mesh centre; i is local to the chunk at qbase
__global__ void batch_query_morton_kernel(const float* __restrict__ pts, int64_t n, int64_t qbase,
                                          const int64_t* __restrict__ qoff, int nmesh,
                                          const float* __restrict__ bounds, int bits, uint32_t* __restrict__ keys,
                                          uint32_t* __restrict__ vals) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int m = segment_of64(qoff, nmesh, qbase + i);
  const float* b = bounds + 6 * (int64_t)m;
  float emax = fmaxf(b[3] - b[0], fmaxf(b[4] - b[1], b[5] - b[2]));
  emax = emax > 0.f ? emax : 1.f;
  const float qmax = (float)((1u << bits) - 1u);
  const float inv = qmax / (2.0f * emax);
  const float q[3] = {(pts[3 * i] - (0.5f * (b[0] + b[3]) - emax)) * inv,
                      (pts[3 * i + 1] - (0.5f * (b[1] + b[4]) - emax)) * inv,
                      (pts[3 * i + 2] - (0.5f * (b[2] + b[5]) - emax)) * inv};
  uint32_t code = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float t = fminf(fmaxf(q[a], 0.f), qmax);
    if (!(t == t)) t = 0.f;
    code |= (uint32_t)spread3_21((uint64_t)t) << a;
  }
  keys[i] = ((uint32_t)m << (3 * bits)) | code;
  vals[i] = (uint32_t)i;
}

int mesh_bits(int nmesh) {
  int mbits = 0;
  while ((1ll << mbits) < nmesh) ++mbits;
  return mbits;
}

size_t batch_udf_bytes(int64_t n) {
  const int64_t c = n < kBatchChunk ? (n > 0 ? n : 1) : kBatchChunk;
  Workspace ws(nullptr, 0);
  UdfWs w;
  const size_t base = carve_udf(w, ws, c, A3D_UDF_SORT_QUERIES);
  return base + (size_t)spill_owner_bound(c) * kSpillCap * sizeof(uint2) + 512;
}

// like: the size of the call whose order and kernel are used (0: this one's own,
// launch by launch); the autotuner times its samples with those of the whole call
int batch_udf(const a3d_bvh_batch* bvh, const void* children, int64_t num_children, const float* points,
              const int64_t* qoff, int64_t n, int64_t like, float* distances, int32_t* face_ids, float* closest_points,
              float* uvw, TaskShape shape, unsigned long long* stats,
              void* workspace, size_t workspace_bytes, cudaStream_t s) {
  A3D_REQUIRE(bvh && bvh->nodes && bvh->tris && bvh->roots && bvh->bounds && bvh->num_meshes > 0 &&
                  bvh->num_faces > 0 && bvh->num_faces < (1ll << 28),
              A3D_ERR_ARGUMENT, "batch_udf: invalid batch");
  A3D_REQUIRE(n >= 0 && n < (1ll << 40), A3D_ERR_ARGUMENT, "batch_udf: bad number of queries");
  A3D_REQUIRE(((uintptr_t)children & 31) == 0, A3D_ERR_ARGUMENT, "batch_udf: child records must be 32-B aligned");
  A3D_REQUIRE(workspace, A3D_ERR_WORKSPACE, "batch_udf: no workspace");
  const int mbits = mesh_bits(bvh->num_meshes);
  A3D_REQUIRE(mbits <= 26, A3D_ERR_ARGUMENT, "batch_udf: too many meshes");
  int bits = (32 - mbits) / 3;
  bits = bits < 10 ? bits : 10;
  const int64_t c = n < kBatchChunk ? (n > 0 ? n : 1) : kBatchChunk;
  Workspace ws(workspace, workspace_bytes);
  UdfWs w;
  carve_udf(w, ws, c, A3D_UDF_SORT_QUERIES);
  A3D_REQUIRE(ws.ok(), A3D_ERR_WORKSPACE, "batch_udf: workspace too small");
  {
    const uintptr_t base = ((uintptr_t)workspace + ws.used + 255) & ~(uintptr_t)255;
    const uintptr_t endp = (uintptr_t)workspace + workspace_bytes;
    const int64_t owners = base < endp ? (int64_t)((endp - base) / (kSpillCap * sizeof(uint2))) : 0;
    w.spill = owners > 0 ? (uint2*)base : nullptr;
    w.spill_owners = owners;
  }
  A3D_CUDA_TRY(cudaMemsetAsync(w.nrerun, 0, kStatusWords * sizeof(uint32_t), s));
  if (n == 0) return A3D_OK;
  A3D_REQUIRE(points && qoff && distances && face_ids && closest_points, A3D_ERR_ARGUMENT, "batch_udf: null pointer");
  // the node count is only known on the device: guard with the capacity
  const TreeT<true> T{(const WideNode*)bvh->nodes, (const TriRec*)bvh->tris, (uint32_t)bvh->num_faces,
                      (uint32_t)bvh->num_faces, w.nrerun + 3, ChildRecs(children, num_children),
                      children != nullptr ? (uint32_t)num_children : 0u};
  const SignArgs sg{nullptr, nullptr, nullptr, nullptr, nullptr};
  for (int64_t base = 0; base < n; base += kBatchChunk) {
    const int64_t cn = n - base < kBatchChunk ? n - base : kBatchChunk;
    const int64_t as = like > 0 ? like : cn;
    const float* pts = points + 3 * base;
    const uint32_t* perm = nullptr;  // the caller's order (mesh by mesh) when there are few
    if (sorted_queries(T.num_children > 0u, as)) {
      A3D_PDL(batch_query_morton_kernel, dim3((unsigned)ceil_div(cn, 256)), dim3(256), 0, s, pts, cn, base, qoff,
              bvh->num_meshes, bvh->bounds, bits, w.keys, w.vals);
      bool alt = false;
      A3D_TRY(radix_sort_pairs<uint32_t>(w.keys, w.vals, w.keys_alt, w.vals_alt, cn, 0, 3 * bits + mbits,
                                         w.rs_scratch, &alt, s));
      perm = alt ? w.vals_alt : w.vals;
    }
    // per chunk: the re-run list and the pool counter start at zero
    A3D_CUDA_TRY(cudaMemsetAsync(w.nrerun, 0, sizeof(uint32_t), s));
    A3D_CUDA_TRY(cudaMemsetAsync(w.nrerun + 2, 0, sizeof(uint32_t), s));
    const QueryOut out{distances + base, face_ids + base, closest_points + 3 * base, uvw ? uvw + 3 * base : nullptr};
    const MeshSel sel{qoff, bvh->roots, bvh->num_meshes, base};
    if (stats)
      A3D_TRY((launch_udf<false, true, true>(T, pts, cn, as, perm, true, nullptr, out, sg, stats, w, kSeedReuse, sel,
                                             shape, s)));
    else
      A3D_TRY((launch_udf<false, false, true>(T, pts, cn, as, perm, true, nullptr, out, sg, stats, w, kSeedReuse, sel,
                                              shape, s)));
  }
  if (stats) A3D_CUDA_TRY(cudaMemcpyAsync(stats + 2, w.nrerun + 4, sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
  return A3D_OK;
}

// every stride-th query, with the offsets of the sample per mesh
__global__ void sample_queries_kernel(const float* __restrict__ pts, int64_t stride, const int64_t* __restrict__ qoff,
                                      int nmesh, float* __restrict__ spts, int64_t ns, int64_t* __restrict__ sqoff) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ns) {
    const int64_t j = i * stride;
    spts[3 * i] = pts[3 * j];
    spts[3 * i + 1] = pts[3 * j + 1];
    spts[3 * i + 2] = pts[3 * j + 2];
  }
  if (i <= nmesh) sqoff[i] = (qoff[i] + stride - 1) / stride;  // first sample at or after qoff[i]
}

struct TuneWs {
  float* pts;
  int64_t* qoff;
  float* dist;
  int32_t* fid;
  float* cp;
  void* udf_ws;
  size_t udf_bytes;
};

size_t carve_tune(TuneWs& t, Workspace& ws, int64_t ns, int nmesh) {
  t.pts = ws.take<float>(3 * ns);
  t.qoff = ws.take<int64_t>(nmesh + 1);
  t.dist = ws.take<float>(ns);
  t.fid = ws.take<int32_t>(ns);
  t.cp = ws.take<float>(3 * ns);
  t.udf_bytes = batch_udf_bytes(ns);
  t.udf_ws = ws.take<unsigned char>((int64_t)t.udf_bytes);
  return ws.used;
}

}  // namespace
}  // namespace a3d

extern "C" int a3d_udf_status(const void* workspace, uint32_t* status_out, a3d_stream_t stream) {
  A3D_REQUIRE(workspace && status_out, A3D_ERR_ARGUMENT, "udf_status: null pointer");
  uint32_t w[a3d::kStatusWords];
  A3D_CUDA_TRY(cudaMemcpyAsync(w, workspace, sizeof(w), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
  A3D_CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
  status_out[0] = w[4];  // queries re-run by the deep-stack kernel
  status_out[1] = w[1];  // deep-stack overflow
  status_out[2] = 0u;
  status_out[3] = w[3];  // guard faults
  return A3D_OK;
}

extern "C" size_t a3d_batch_udf_workspace_bytes(int64_t num_queries, int32_t num_meshes) {
  (void)num_meshes;
  return a3d::batch_udf_bytes(num_queries);
}

extern "C" int a3d_batch_udf(const a3d_bvh_batch* bvh, const float* points, const int64_t* query_offsets,
                             int64_t num_queries, float* distances, int32_t* face_ids, float* closest_points,
                             float* uvw, const a3d_udf_tuning* tuning, unsigned long long* stats, void* workspace,
                             size_t workspace_bytes, a3d_stream_t stream) {
  return a3d_batch_udf_children(bvh, nullptr, 0, points, query_offsets, num_queries, distances, face_ids,
                                closest_points, uvw, tuning, stats, workspace, workspace_bytes, stream);
}

extern "C" int a3d_batch_udf_children(const a3d_bvh_batch* bvh, const void* children, int64_t num_children,
                                      const float* points, const int64_t* query_offsets, int64_t num_queries,
                                      float* distances, int32_t* face_ids, float* closest_points, float* uvw,
                                      const a3d_udf_tuning* tuning, unsigned long long* stats, void* workspace,
                                      size_t workspace_bytes, a3d_stream_t stream) {
  A3D_REQUIRE(num_children >= 0 && num_children < (1ll << 31), A3D_ERR_ARGUMENT, "batch_udf: bad child-record count");
  a3d::TaskShape shape{0, 0};
  if (tuning) {
    A3D_REQUIRE(tuning->pool >= 0 && tuning->pool <= 4096 && tuning->blocks_per_sm >= 0, A3D_ERR_ARGUMENT,
                "batch_udf: bad tuning");
    if (tuning->pool > 0) shape.pool = tuning->pool;
    shape.blocks_per_sm = tuning->blocks_per_sm;
  }
  return a3d::batch_udf(bvh, children, num_children, points, query_offsets, num_queries, 0, distances, face_ids,
                        closest_points, uvw, shape, stats, workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" size_t a3d_batch_autotune_workspace_bytes(int64_t sample_queries, int32_t num_meshes) {
  a3d::Workspace ws(nullptr, 0);
  a3d::TuneWs t;
  return a3d::carve_tune(t, ws, sample_queries > 0 ? sample_queries : 1, num_meshes > 0 ? num_meshes : 1) + 256;
}

extern "C" int a3d_batch_autotune(const a3d_bvh_batch* bvh, const float* points, const int64_t* query_offsets,
                                  int64_t num_queries, int64_t sample_queries, void* workspace,
                                  size_t workspace_bytes, a3d_udf_tuning* best, float* best_ms,
                                  a3d_stream_t stream) {
  return a3d_batch_autotune_children(bvh, nullptr, 0, points, query_offsets, num_queries, sample_queries, workspace,
                                  workspace_bytes, best, best_ms, stream);
}

extern "C" int a3d_batch_autotune_children(const a3d_bvh_batch* bvh, const void* children, int64_t num_children,
                                        const float* points, const int64_t* query_offsets, int64_t num_queries,
                                        int64_t sample_queries, void* workspace, size_t workspace_bytes,
                                        a3d_udf_tuning* best, float* best_ms, a3d_stream_t stream_) {
  using namespace a3d;
  cudaStream_t s = (cudaStream_t)stream_;
  A3D_REQUIRE(bvh && points && query_offsets && best && num_queries > 0 && sample_queries > 0, A3D_ERR_ARGUMENT,
              "batch_autotune: bad argument");
  A3D_REQUIRE(sample_queries <= kBatchChunk, A3D_ERR_ARGUMENT, "batch_autotune: sample larger than one launch");
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  A3D_CUDA_TRY(cudaStreamIsCapturing(s, &cap));
  A3D_REQUIRE(cap == cudaStreamCaptureStatusNone, A3D_ERR_ARGUMENT,
              "batch_autotune: times launches on the host; call it outside stream capture");
  const int64_t stride = (num_queries + sample_queries - 1) / sample_queries;
  const int64_t ns = (num_queries + stride - 1) / stride;
  Workspace ws(workspace, workspace_bytes);
  TuneWs t;
  carve_tune(t, ws, ns, bvh->num_meshes);
  A3D_REQUIRE(workspace && ws.ok(), A3D_ERR_WORKSPACE, "batch_autotune: workspace too small");
  const int64_t th = ns > (int64_t)bvh->num_meshes + 1 ? ns : (int64_t)bvh->num_meshes + 1;
  A3D_PDL(sample_queries_kernel, dim3((unsigned)ceil_div(th, 256)), dim3(256), 0, s, points, stride, query_offsets,
          bvh->num_meshes, t.pts, ns, t.qoff);
  // order and kernel of the call that is tuned for (of its first launch), and the
  // blocks of that kernel an SM holds
  const int64_t like = num_queries < kBatchChunk ? num_queries : kBatchChunk;
  const bool records = children != nullptr && num_children > 0, two = two_lanes(records, like);
  int occ = 0;
  A3D_TRY((records && two ? group_blocks_per_sm<2, true, false, true>(&occ)
           : records      ? group_blocks_per_sm<4, true, false, true>(&occ)
           : two          ? group_blocks_per_sm<2, false, false, true>(&occ)
                          : group_blocks_per_sm<4, false, false, true>(&occ)));
  const int pools[4] = {32, 64, 128, 256};
  const int bpss[3] = {occ, occ * 3 / 4, occ / 2};
  cudaEvent_t e0, e1;
  A3D_CUDA_TRY(cudaEventCreate(&e0));
  A3D_CUDA_TRY(cudaEventCreate(&e1));
  float best_t = INFINITY;
  a3d_udf_tuning bt{64, kAllBlocks, 0, 0};
  int rc = A3D_OK;
  for (int pi = 0; pi < 4 && rc == A3D_OK; ++pi) {
    for (int bi = 0; bi < 3 && rc == A3D_OK; ++bi) {
      const int bps = bpss[bi];
      if (bps < 1 || (bi > 0 && bps == bpss[bi - 1])) continue;
      const TaskShape shape{pools[pi], bps};
      // one warm-up run, then two timed
      for (int rep = 0; rep < 3 && rc == A3D_OK; ++rep) {
        if (rep == 1 && cudaEventRecord(e0, s) != cudaSuccess) rc = A3D_ERR_CUDA;
        if (rc == A3D_OK)
          rc = batch_udf(bvh, children, num_children, t.pts, t.qoff, ns, like, t.dist, t.fid, t.cp, nullptr, shape,
                         nullptr, t.udf_ws, t.udf_bytes, s);
      }
      float ms = 0.f;
      if (rc == A3D_OK && (cudaEventRecord(e1, s) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
                           cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess))
        rc = A3D_ERR_CUDA;
      if (rc != A3D_OK) break;
      ms *= 0.5f;
      if (ms < best_t) {
        best_t = ms;
        bt = a3d_udf_tuning{pools[pi], bi == 0 ? kAllBlocks : bps, 0, 0};
      }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc != A3D_OK) return rc;
  *best = bt;
  if (best_ms) *best_ms = best_t;
  return A3D_OK;
}
