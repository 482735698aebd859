// Ray queries over the wide BVH: nearest hit, all hits, ray-parity inside
// votes.
//
// Replaces bvh_ray_intersect_kernel and bvh_ray_all_hit_kernel
// (atom3d/kernels/bvh_kernels.cu:469-553, :935-1022) and the host-side
// coalescing / vote loop of MeshBVH._sdf_parity and _signed_crossing_count
// (atom3d/core/mesh_bvh.py:850-948), which here is one fused kernel.
//
// The per-triangle maths is the reference's (Triangle::ray_intersect,
// ::normal, ::barycentric at bvh_kernels.cu:89-221) restated operation by
// operation with round-to-nearest intrinsics, so t values, hit decisions and
// signs are bit-identical to the oracle's restatement.  Child boxes are the
// outward-rounded quantised ones and a box is skipped only when its entry
// distance exceeds the current bound by a relative 2e-6, so pruning never
// drops a hit.  A triangle miss is +inf (the reference uses a 1e10 sentinel,
// which a max_t above 1e10 would count as a hit).
#include <float.h>
#include <math.h>

#include "bvh_layout.cuh"
#include "primitives.cuh"

namespace a3d {

namespace {

constexpr int kRayThreads = 128;
// shared-memory stack entries per ray; a ray that needs more is re-run with a
// deep local stack
constexpr int kRayShared = 20;
constexpr int kRayDeep = 256;    // local-memory stack of the re-run kernel
constexpr int kAllDepth = 192;   // node stack of the all-hit traversals
constexpr int kParityCap = 256;  // hits per (point, direction) kept by the parity kernel
constexpr float kPruneSlack = 1.000002f;

// The largest entry distance of a box that can hold a hit before t.  Finite: a
// missed child and an empty slot, whose reference names nothing, have the entry
// distance +inf, which no t admits.
__device__ __forceinline__ float prune_limit(float t) { return fminf(t * kPruneSlack, FLT_MAX); }

struct V3 {
  float x, y, z;
};

__device__ __forceinline__ V3 ld3(const float* p, int64_t i) { return V3{p[3 * i], p[3 * i + 1], p[3 * i + 2]}; }
__device__ __forceinline__ V3 vsub(V3 a, V3 b) {
  return V3{__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)};
}
__device__ __forceinline__ float vdot(V3 a, V3 b) {
  return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ V3 vcross(V3 a, V3 b) {
  return V3{__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y)), __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z)),
            __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x))};
}
__device__ __forceinline__ V3 vpoint(V3 o, V3 d, float t) {
  return V3{__fadd_rn(o.x, __fmul_rn(d.x, t)), __fadd_rn(o.y, __fmul_rn(d.y, t)), __fadd_rn(o.z, __fmul_rn(d.z, t))};
}

struct Tri {
  V3 a, b, c;
  int32_t face;
};

__device__ __forceinline__ Tri load_tri(const TriRec* __restrict__ tris, uint32_t i) {
  const float4* p = reinterpret_cast<const float4*>(tris + i);
  const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
  return Tri{V3{a.x, a.y, a.z}, V3{b.x, b.y, b.z}, V3{c.x, c.y, c.z}, __float_as_int(a.w)};
}

// Moller-Trumbore as Triangle::ray_intersect; +inf for a miss
__device__ __forceinline__ float ray_tri(const Tri& t, V3 ro, V3 rd) {
  const double eps_edge = 1.19209290e-7;
  const V3 e1 = vsub(t.b, t.a), e2 = vsub(t.c, t.a);
  const V3 h = vcross(rd, e2);
  const float det = vdot(e1, h);
  const float ad = fabsf(det);
  if (ad < 1e-8f) return INFINITY;
  // Nearly every triangle tested is missed, most of them clearly: u and v
  // against |det| with margins far above the rounding of f and the products,
  // before the divide and the FP64 comparisons that decide the rest.  (An
  // overflow to inf or NaN passes no rejection that the exact test would not
  // make.)
  const V3 s = vsub(ro, t.a);
  const float su = vdot(s, h);
  const float au = det < 0.f ? -su : su;
  if (au < -1e-5f * ad || au > 1.00001f * ad) return INFINITY;
  const V3 q = vcross(s, e1);
  const float sv = vdot(rd, q);
  const float av = det < 0.f ? -sv : sv;
  if (av < -1e-5f * ad || av > 1.00001f * ad) return INFINITY;
  const float f = __fdiv_rn(1.0f, det);
  const double u = __dmul_rn((double)f, (double)su);
  if (u < -eps_edge || u > 1.0 + eps_edge) return INFINITY;
  const double v = __dmul_rn((double)f, (double)sv);
  if (v < -eps_edge || __dadd_rn(u, v) > 1.0 + eps_edge) return INFINITY;
  const float tt = __fmul_rn(f, vdot(e2, q));
  return tt > 1e-8f ? tt : INFINITY;
}

// Triangle::normal: unit normal of (b - a) x (c - a), (0, 0, 1) if degenerate
__device__ __forceinline__ V3 tri_normal(const Tri& t) {
  const V3 n = vcross(vsub(t.b, t.a), vsub(t.c, t.a));
  const float len = __fsqrt_rn(vdot(n, n));
  if (len > 1e-10f) {
    const float inv = __fdiv_rn(1.0f, len);
    return V3{__fmul_rn(n.x, inv), __fmul_rn(n.y, inv), __fmul_rn(n.z, inv)};
  }
  return V3{0.f, 0.f, 1.f};
}

// barycentrics of a point on the triangle: floor `dfloor` on the
// denominator (Triangle::barycentric, 1e-10) or additive `dadd`
// (MeshBVH._bary_from_hit, 1e-12)
__device__ __forceinline__ V3 tri_bary(const Tri& t, V3 p, bool additive) {
  const V3 v0 = vsub(t.b, t.a), v1 = vsub(t.c, t.a), v2 = vsub(p, t.a);
  const float d00 = vdot(v0, v0), d01 = vdot(v0, v1), d11 = vdot(v1, v1), d20 = vdot(v2, v0), d21 = vdot(v2, v1);
  float denom = __fsub_rn(__fmul_rn(d00, d11), __fmul_rn(d01, d01));
  denom = additive ? __fadd_rn(denom, 1e-12f) : fmaxf(denom, 1e-10f);
  const float v = __fdiv_rn(__fsub_rn(__fmul_rn(d11, d20), __fmul_rn(d01, d21)), denom);
  const float w = __fdiv_rn(__fsub_rn(__fmul_rn(d00, d21), __fmul_rn(d01, d20)), denom);
  return V3{__fsub_rn(__fsub_rn(1.0f, v), w), v, w};
}

struct Ray {
  V3 o, d, inv;
};

__device__ __forceinline__ Ray make_ray(V3 o, V3 d) {
  auto safe = [](float x) { return fabsf(x) > 1e-8f ? x : (x >= 0.f ? 1e-8f : -1e-8f); };
  return Ray{o, d, V3{__fdiv_rn(1.0f, safe(d.x)), __fdiv_rn(1.0f, safe(d.y)), __fdiv_rn(1.0f, safe(d.z))}};
}

// entry distances of a node's four children (+inf for a miss or an empty
// slot) and their references
__device__ __forceinline__ void child_entries(const WideNode* __restrict__ nodes, uint32_t ref, const Ray& r,
                                              float* tc, uint32_t* rc) {
  const int4* np = reinterpret_cast<const int4*>(nodes + ref);
  int4 w0, w1, w2, w3;
  ldg256(np, w0, w1);
  ldg256(np + 2, w2, w3);
  const float ox = __int_as_float(w0.x), oy = __int_as_float(w0.y), oz = __int_as_float(w0.z);
  const uint32_t meta = (uint32_t)w0.w;
  const float sx = __uint_as_float((meta & 0xffu) << 23);
  const float sy = __uint_as_float(((meta >> 8) & 0xffu) << 23);
  const float sz = __uint_as_float(((meta >> 16) & 0xffu) << 23);
  const int nch = (int)(meta >> 24);
  rc[0] = (uint32_t)w2.z;
  rc[1] = (uint32_t)w2.w;
  rc[2] = (uint32_t)w3.x;
  rc[3] = (uint32_t)w3.y;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float lx = dequant((uint32_t)w1.x, c, sx, ox), ly = dequant((uint32_t)w1.y, c, sy, oy);
    const float lz = dequant((uint32_t)w1.z, c, sz, oz), hx = dequant((uint32_t)w1.w, c, sx, ox);
    const float hy = dequant((uint32_t)w2.x, c, sy, oy), hz = dequant((uint32_t)w2.y, c, sz, oz);
    float t1 = (lx - r.o.x) * r.inv.x, t2 = (hx - r.o.x) * r.inv.x;
    float tmin = fminf(t1, t2), tmax = fmaxf(t1, t2);
    t1 = (ly - r.o.y) * r.inv.y;
    t2 = (hy - r.o.y) * r.inv.y;
    tmin = fmaxf(tmin, fminf(t1, t2));
    tmax = fminf(tmax, fmaxf(t1, t2));
    t1 = (lz - r.o.z) * r.inv.z;
    t2 = (hz - r.o.z) * r.inv.z;
    tmin = fmaxf(tmin, fminf(t1, t2));
    tmax = fminf(tmax, fmaxf(t1, t2));
    tc[c] = (c < nch && tmax >= tmin && tmax >= 0.f) ? fmaxf(tmin, 0.f) : INFINITY;
  }
}

__device__ __forceinline__ void cswap(float& ta, uint32_t& ra, float& tb, uint32_t& rb) {
  if (tb < ta || (tb == ta && rb < ra)) {
    const float t = ta;
    ta = tb;
    tb = t;
    const uint32_t x = ra;
    ra = rb;
    rb = x;
  }
}

struct LocalStack {
  uint2 s[kRayDeep];
  int sp;
  static constexpr int kDepth = kRayDeep;
  __device__ __forceinline__ void push(uint32_t ref, float t) { s[sp++] = make_uint2(ref, __float_as_uint(t)); }
  __device__ __forceinline__ uint2 pop() { return s[--sp]; }
};

// Nearest hit: children in ascending entry distance, strict "<" on t.
// Returns false when the stack would overflow (the ray is re-run).
template <typename Stack>
__device__ bool nearest(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris, const Ray& r,
                        float& mint, uint32_t& best, Stack& st) {
  uint32_t ref = 0;
  bool have = true;
  for (;;) {
    if (have) {
      if (!ref_is_leaf(ref)) {
        float tc[4];
        uint32_t rc[4];
        child_entries(nodes, ref, r, tc, rc);
        cswap(tc[0], rc[0], tc[1], rc[1]);
        cswap(tc[2], rc[2], tc[3], rc[3]);
        cswap(tc[0], rc[0], tc[2], rc[2]);
        cswap(tc[1], rc[1], tc[3], rc[3]);
        cswap(tc[1], rc[1], tc[2], rc[2]);
        const float lim = prune_limit(mint);
        int q = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) q += tc[c] <= lim ? 1 : 0;
        if (q > 0) {
          if (st.sp + (q - 1) > Stack::kDepth) return false;
#pragma unroll
          for (int c = 3; c >= 1; --c)
            if (c < q) st.push(rc[c], tc[c]);
          ref = rc[0];
          continue;
        }
      } else {
        const uint32_t f0 = leaf_first(ref), cnt = leaf_count(ref);
        for (uint32_t i = 0; i < cnt; ++i) {
          const float t = ray_tri(load_tri(tris, f0 + i), r.o, r.d);
          if (t < mint) {
            mint = t;
            best = f0 + i;
          }
        }
      }
    }
    have = false;
    while (st.sp > 0) {
      const uint2 e = st.pop();
      if (__uint_as_float(e.y) <= mint * kPruneSlack) {
        ref = e.x;
        have = true;
        break;
      }
    }
    if (!have) return true;
  }
}

struct RayOut {
  uint8_t* hit;
  float* t;
  int32_t* face;
  float* point;
  float* normal;
  float* uvw;
};

// The nearest-hit traversal: one ray a lane, persistent warps that hand new
// rays to lanes as they finish.  A warp alternates node steps, while at least
// kNodeLanes of its rays are at an inner node, with one leaf step in which the
// triangles of all rays at a leaf are spread evenly over the lanes.  The order
// of each ray's visits is that of nearest().  Writes each ray's t and, for
// ray_finish_kernel, the triangle's record in place of the face.
// Bound by its instructions: with a ray a thread from start to end, node and
// leaf in one loop and the divide and FP64 comparisons on every triangle, 7 of
// 32 lanes were active and 4.2M rays (half a camera's, half scattered) took
// 2.00 ms; now 0.96.
constexpr int kRayWarps = kRayThreads / 32;
// rays at a node below which a warp turns to its leaves, resident blocks an SM,
// most rays a warp takes at a time (4.2M rays, 1.31M triangles: 1066, 1024,
// 1008 and 1010 us at 12, 16, 20 and 24 lanes; pools of 128 / 64 / 32: 1012 /
// 961 / 966 us at 8 blocks)
constexpr int kNodeLanes = 20;
constexpr int kRayBlocks = 8;
constexpr int kParityBlocks = 7;
constexpr int64_t kRayPool = 64;
constexpr int kTriRow = 33;  // results at position-in-leaf * 33 + owner: distinct banks
constexpr uint32_t kNoItem = 0xffffffffu;  // no node or leaf; no reference has this value

struct RaySmem {
  uint2 stack[kRayShared][32];
  uint2 own[32];  // a leaf step's rays in lane order: first triangle less its first task, lane | first task << 8
  float trid[kMaxLeafTris * kTriRow];
};

__global__ void __launch_bounds__(kRayThreads, kRayBlocks)
    ray_nearest_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                       const float* __restrict__ ro, const float* __restrict__ rd, uint32_t n, float max_t,
                       float* __restrict__ t_out, int32_t* __restrict__ tri_out, uint32_t* __restrict__ rerun,
                       uint32_t* __restrict__ nrerun, uint32_t* __restrict__ pool_counter, uint32_t pool) {
  pdl_wait();
  __shared__ RaySmem smem[kRayWarps];
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  RaySmem& S = smem[threadIdx.x >> 5];
  uint32_t pos = 0, end = 0;
  bool exhausted = false;
  bool live = false;
  uint32_t i = 0, ref = kNoItem, best = 0xffffffffu;
  float mint = max_t;
  int sp = 0;
  Ray r{};

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
      const uint32_t rank = __popc(want & ((1u << lane) - 1u));
      const bool mine = ((want >> lane) & 1u) && rank < take;
      if (mine) {
        i = pos + rank;
        r = make_ray(ld3(ro, i), ld3(rd, i));
        mint = max_t;
        best = 0xffffffffu;
        sp = 0;
        ref = 0u;
        live = true;
      }
      pos += take;
      want &= ~__ballot_sync(FULL, mine);
    }
  };
  auto pop = [&]() {
    ref = kNoItem;
    while (sp > 0) {
      --sp;
      const uint2 e = S.stack[sp][lane];
      if (__uint_as_float(e.y) <= mint * kPruneSlack) {
        ref = e.x;
        break;
      }
    }
  };

  distribute(FULL);
  while (__any_sync(FULL, live)) {
    // (a) node steps
    for (;;) {
      const unsigned at_node = __ballot_sync(FULL, (int)ref >= 0);
      if (__popc(at_node) < kNodeLanes &&
          (at_node == 0u || __any_sync(FULL, live && (int)ref < 0)))
        break;
      if ((int)ref >= 0) {
        float tc[4];
        uint32_t rc[4];
        child_entries(nodes, ref, r, tc, rc);
        cswap(tc[0], rc[0], tc[1], rc[1]);
        cswap(tc[2], rc[2], tc[3], rc[3]);
        cswap(tc[0], rc[0], tc[2], rc[2]);
        cswap(tc[1], rc[1], tc[3], rc[3]);
        cswap(tc[1], rc[1], tc[2], rc[2]);
        const float lim = prune_limit(mint);
        int q = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) q += tc[c] <= lim ? 1 : 0;
        if (q == 0) {
          pop();
        } else if (sp + (q - 1) > kRayShared) {
          rerun[atomicAdd(nrerun, 1u)] = i;  // no room: re-run with a deep stack
          live = false;
          ref = kNoItem;
        } else {
#pragma unroll
          for (int c = 3; c >= 1; --c)
            if (c < q) S.stack[sp++][lane] = make_uint2(rc[c], __float_as_uint(tc[c]));
          ref = rc[0];
        }
      }
    }
    // (b) leaf step
    const uint32_t cnt = live && (int)ref < 0 && ref != kNoItem ? leaf_count(ref) : 0u;
    const unsigned owners = __ballot_sync(FULL, cnt > 0u);
    if (owners) {
      const unsigned lt = (1u << lane) - 1u;
      uint32_t off = 0, total = 0;  // first task of this lane, tasks in all
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const unsigned m = __ballot_sync(FULL, (cnt >> b) & 1u);
        off += (uint32_t)__popc(m & lt) << b;
        total += (uint32_t)__popc(m) << b;
      }
      if (cnt > 0u) S.own[__popc(owners & lt)] = make_uint2(leaf_first(ref) - off, (uint32_t)lane | (off << 8));
      __syncwarp();
      int before = -1;  // owners whose first task lies before this group of 32
      for (uint32_t t0 = 0; t0 < total; t0 += 32) {
        const unsigned firsts = __reduce_or_sync(FULL, cnt > 0u && (off >> 5) == (t0 >> 5) ? 1u << (off & 31u) : 0u);
        const uint2 w = S.own[before + __popc(firsts & (0xffffffffu >> (31 - lane)))];
        before += __popc(firsts);
        const int o = (int)(w.y & 31u);
        const V3 qo{__shfl_sync(FULL, r.o.x, o), __shfl_sync(FULL, r.o.y, o), __shfl_sync(FULL, r.o.z, o)};
        const V3 qd{__shfl_sync(FULL, r.d.x, o), __shfl_sync(FULL, r.d.y, o), __shfl_sync(FULL, r.d.z, o)};
        const uint32_t t = t0 + (uint32_t)lane;
        if (t < total) S.trid[(t - (w.y >> 8)) * kTriRow + o] = ray_tri(load_tri(tris, w.x + t), qo, qd);
      }
      __syncwarp();
      if (cnt > 0u) {
        const uint32_t f0 = leaf_first(ref);
        for (uint32_t k = 0; k < cnt; ++k) {
          const float t = S.trid[k * kTriRow + lane];
          if (t < mint) {
            mint = t;
            best = f0 + k;
          }
        }
        pop();
      }
      __syncwarp();
    }
    // (c) finished rays, new ones
    const bool done = live && ref == kNoItem;
    if (done) {
      t_out[i] = mint;
      tri_out[i] = (int32_t)best;
      live = false;
    }
    const unsigned free_lanes = __ballot_sync(FULL, !live);
    if (!exhausted || pos < end) distribute(free_lanes);
  }
}

__global__ void __launch_bounds__(64)
    ray_nearest_rerun_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                             const float* __restrict__ ro, const float* __restrict__ rd, float max_t,
                             float* __restrict__ t_out, int32_t* __restrict__ tri_out,
                             const uint32_t* __restrict__ rerun, const uint32_t* __restrict__ nrerun,
                             uint32_t* __restrict__ overflow) {
  pdl_wait();
  const uint32_t m = *nrerun;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = rerun[k];
    const Ray r = make_ray(ld3(ro, i), ld3(rd, i));
    float mint = max_t;
    uint32_t best = 0xffffffffu;
    LocalStack st;
    st.sp = 0;
    if (!nearest(nodes, tris, r, mint, best, st)) atomicExch(overflow, 1u);
    t_out[i] = mint;
    tri_out[i] = (int32_t)best;
  }
}

// the outputs of ray i but t, for the nearest hit (t, best)
__device__ __forceinline__ void write_ray(const TriRec* __restrict__ tris, const float* __restrict__ face_normals,
                                          V3 o, V3 d, int64_t i, float t, uint32_t best, const RayOut& out) {
  const bool hit = best != 0xffffffffu;
  out.hit[i] = hit ? 1 : 0;
  V3 p{0.f, 0.f, 0.f}, nrm{0.f, 0.f, 0.f}, bc{0.f, 0.f, 0.f};
  int32_t face = -1;
  if (hit) {
    const Tri tr = load_tri(tris, best);
    face = tr.face;
    p = vpoint(o, d, t);
    if (out.uvw) bc = tri_bary(tr, p, true);
    if (face_normals) nrm = ld3(face_normals, face);
  }
  out.face[i] = face;
  if (out.point) {
    out.point[3 * i] = p.x;
    out.point[3 * i + 1] = p.y;
    out.point[3 * i + 2] = p.z;
  }
  if (out.normal) {
    out.normal[3 * i] = nrm.x;
    out.normal[3 * i + 1] = nrm.y;
    out.normal[3 * i + 2] = nrm.z;
  }
  if (out.uvw) {
    out.uvw[3 * i] = bc.x;
    out.uvw[3 * i + 1] = bc.y;
    out.uvw[3 * i + 2] = bc.z;
  }
}

// The remaining outputs of each ray; out.t holds t and out.face the triangle
// record on entry.
__global__ void __launch_bounds__(256)
    ray_finish_kernel(const TriRec* __restrict__ tris, const float* __restrict__ face_normals,
                      const float* __restrict__ ro, const float* __restrict__ rd, int64_t n, RayOut out) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  write_ray(tris, face_normals, ld3(ro, i), ld3(rd, i), i, out.t[i], (uint32_t)out.face[i], out);
}

// A whole ray a thread, outputs included, for trees of one node (up to some 24
// triangles): a walk is the root and at most four leaves, and the hand-over
// between lanes and two more passes cost more than lanes that wait.  us a call,
// three passes / this, 300,000 and 2M rays: one triangle 48 / 40 and 97 / 75, a
// cube's twelve 61 / 53 and 161 / 152, twenty of a sphere 64 / 57 and 161 / 167;
// with three nodes (a cube of 48) 72 / 79 and 192 / 285.
constexpr int64_t kRayWholeNodes = 1;

__global__ void __launch_bounds__(kRayThreads)
    ray_whole_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                         const float* __restrict__ face_normals, const float* __restrict__ ro,
                         const float* __restrict__ rd, int64_t n, float max_t, RayOut out,
                         uint32_t* __restrict__ overflow) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * kRayThreads + threadIdx.x;
  if (i >= n) return;
  const Ray r = make_ray(ld3(ro, i), ld3(rd, i));
  float mint = max_t;
  uint32_t best = 0xffffffffu;
  LocalStack st;
  st.sp = 0;
  if (!nearest(nodes, tris, r, mint, best, st)) atomicExch(overflow, 1u);
  out.t[i] = mint;
  write_ray(tris, face_normals, r.o, r.d, i, mint, best, out);
}

// All hits of one ray in traversal order; `emit(t, tri)` for each
// non-grazing hit with 0 < t < max_t.  Returns false on stack overflow.
template <typename Emit>
__device__ bool all_hits(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris, const Ray& r,
                         float max_t, Emit emit) {
  uint32_t stack[kAllDepth];
  int sp = 0;
  stack[sp++] = 0u;
  const float lim = prune_limit(max_t);
  bool ok = true;
  while (sp > 0) {
    const uint32_t ref = stack[--sp];
    if (!ref_is_leaf(ref)) {
      float tc[4];
      uint32_t rc[4];
      child_entries(nodes, ref, r, tc, rc);
#pragma unroll
      for (int c = 3; c >= 0; --c) {
        if (tc[c] <= lim) {
          if (sp < kAllDepth) stack[sp++] = rc[c];
          else ok = false;
        }
      }
    } else {
      const uint32_t f0 = leaf_first(ref), cnt = leaf_count(ref);
      for (uint32_t k = 0; k < cnt; ++k) {
        const Tri t = load_tri(tris, f0 + k);
        const float th = ray_tri(t, r.o, r.d);
        if (th > 0.0f && th < max_t) {
          const float ndotd = vdot(tri_normal(t), r.d);
          if (ndotd > -1e-4f && ndotd < 1e-4f) continue;  // grazing
          emit(th, t, ndotd > 0.0f ? 1 : -1);
        }
      }
    }
  }
  return ok;
}

__global__ void ray_all_count_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                                     const float* __restrict__ ro, const float* __restrict__ rd, int64_t n,
                                     float max_t, int32_t* __restrict__ counts, uint32_t* __restrict__ overflow) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Ray r = make_ray(ld3(ro, i), ld3(rd, i));
  int32_t c = 0;
  if (!all_hits(nodes, tris, r, max_t, [&](float, const Tri&, int) { ++c; })) atomicExch(overflow, 1u);
  counts[i] = c;
}

struct AllOut {
  int32_t* ray;
  float* t;
  int32_t* face;
  int32_t* sign;
  float* point;
  float* uvw;
};

__global__ void ray_all_collect_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                                       const float* __restrict__ ro, const float* __restrict__ rd, int64_t n,
                                       float max_t, const int64_t* __restrict__ offsets, AllOut out) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Ray r = make_ray(ld3(ro, i), ld3(rd, i));
  int64_t w = offsets[i];
  const int64_t wend = offsets[i + 1];
  all_hits(nodes, tris, r, max_t, [&](float th, const Tri& t, int s) {
    if (w >= wend) return;  // the count pass saw the same hits; kept as a bound
    out.ray[w] = (int32_t)i;
    out.t[w] = th;
    out.face[w] = t.face;
    out.sign[w] = s;
    const V3 p = vpoint(r.o, r.d, th);
    if (out.point) {
      out.point[3 * w] = p.x;
      out.point[3 * w + 1] = p.y;
      out.point[3 * w + 2] = p.z;
    }
    if (out.uvw) {
      const V3 b = tri_bary(t, p, false);
      out.uvw[3 * w] = b.x;
      out.uvw[3 * w + 1] = b.y;
      out.uvw[3 * w + 2] = b.z;
    }
    ++w;
  });
}

// Signed crossing count of a ray from its k hits, sorted by t (sign: the hit's
// side): near-coincident hits (|dt| < coalesce) are merged -- a group whose
// hits all share a sign counts as one crossing of that sign, a mixed group as
// (|sum| mod 2) * sign(sum) -- and the ray votes when the count is odd.
template <typename Hit>
__device__ __forceinline__ int parity_vote(int k, float coalesce, Hit hit) {
  int32_t sc = 0;
  int a = 0;
  while (a < k) {
    int b = a + 1;
    float tb;
    int sg;
    hit(a, tb, sg);
    int32_t cnt = 1, sum = sg;
    while (b < k) {
      float t;
      hit(b, t, sg);
      if (!(fabsf(__fsub_rn(t, tb)) < coalesce)) break;
      ++cnt;
      sum += sg;
      tb = t;
      ++b;
    }
    const int32_t sgn = sum > 0 ? 1 : (sum < 0 ? -1 : 0);
    const int32_t asum = sum < 0 ? -sum : sum;
    sc += asum == cnt ? sgn : (asum % 2) * sgn;
    a = b;
  }
  return ((sc < 0 ? -sc : sc) % 2) == 1 ? 1 : 0;
}

// One (direction, point) ray a lane, directions outermost so that a warp's rays
// are parallel; phases as in ray_nearest_kernel, visits in any order.  A ray's
// first hits (t, the sign bit for hits from the front) and stack entries stay in
// shared memory, the rest in local memory; the hits of a ray with more than
// kParityHits are sorted by the whole warp.  votes[i] (zeroed before) counts the
// point's odd rays.  100,000 points, 8 directions, 200,000 triangles: 1.38 ms
// with a thread per point and its directions in turn, 0.55 ms so.
constexpr int kParityHits = 12;
constexpr int kParityStack = 24;

struct ParitySmem {
  uint32_t stack[kParityStack][32];
  float hits[kParityHits][32];
  uint2 own[32];
  float trid[kMaxLeafTris * kTriRow];  // between leaf steps: the hits to sort
  float sorted[kParityCap];
};
static_assert(kMaxLeafTris * kTriRow >= kParityCap, "a ray's hits fit the leaf step's results");

__global__ void __launch_bounds__(kRayThreads, kParityBlocks)
    ray_parity_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                      const float* __restrict__ pts, int64_t n, const float* __restrict__ dirs, int ndir, float max_t,
                      float coalesce, int32_t* __restrict__ votes, uint32_t* __restrict__ overflow,
                      unsigned long long* __restrict__ pool_counter, int64_t pool) {
  pdl_wait();
  __shared__ ParitySmem smem[kRayWarps];
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  ParitySmem& S = smem[threadIdx.x >> 5];
  const int64_t rays = n * ndir;
  const float lim = prune_limit(max_t);
  int64_t pos = 0, end = 0;
  bool exhausted = false, live = false, lost = false;
  int64_t i = 0;
  int dir = 0, sp = 0, nh = 0;
  uint32_t ref = kNoItem;
  Ray r{};
  float more_hits[kParityCap - kParityHits];
  uint32_t more_stack[kAllDepth - kParityStack];

  const uint32_t* deep = more_stack;

  auto pop = [&]() -> uint32_t {
    if (sp == 0) return kNoItem;
    --sp;
    return sp < kParityStack ? S.stack[sp][lane] : deep[sp - kParityStack];
  };
  auto distribute = [&](unsigned want) {
    while (want) {
      if (pos >= end) {
        if (exhausted) break;
        unsigned long long p = 0;
        if (lane == 0) p = atomicAdd(pool_counter, 1ull);
        p = __shfl_sync(FULL, p, 0);
        if (p >= (unsigned long long)ceil_div(rays, pool)) { exhausted = true; break; }
        pos = (int64_t)p * pool;
        end = rays - pos < pool ? rays : pos + pool;
      }
      const int64_t avail = end - pos;
      const int cnt = __popc(want);
      const int take = (int)(avail < cnt ? avail : cnt);
      const int rank = __popc(want & ((1u << lane) - 1u));
      const bool mine = ((want >> lane) & 1u) && rank < take;
      if (mine) {
        const int64_t j = pos + rank;
        dir = (int)(j / n);
        i = j - dir * n;
        r = make_ray(ld3(pts, i), ld3(dirs, dir));
        sp = 0;
        nh = 0;
        ref = 0u;
        live = true;
      }
      pos += take;
      want &= ~__ballot_sync(FULL, mine);
    }
  };

  distribute(FULL);
  while (__any_sync(FULL, live)) {
    // (a) node steps
    for (;;) {
      const unsigned at_node = __ballot_sync(FULL, (int)ref >= 0);
      if (__popc(at_node) < kNodeLanes && (at_node == 0u || __any_sync(FULL, live && (int)ref < 0))) break;
      if ((int)ref >= 0) {
        float tc[4];
        uint32_t rc[4];
        child_entries(nodes, ref, r, tc, rc);
        uint32_t next = kNoItem;
#pragma unroll
        for (int c = 3; c >= 0; --c)
          if (tc[c] <= lim) {
            if (next != kNoItem) {
              if (sp < kParityStack) S.stack[sp++][lane] = next;
              else if (sp < kAllDepth) more_stack[sp++ - kParityStack] = next;
              else lost = true;
            }
            next = rc[c];
          }
        ref = next == kNoItem ? pop() : next;
      }
    }
    // (b) leaf step
    const uint32_t cnt = live && (int)ref < 0 && ref != kNoItem ? leaf_count(ref) : 0u;
    const unsigned owners = __ballot_sync(FULL, cnt > 0u);
    if (owners) {
      const unsigned lt = (1u << lane) - 1u;
      uint32_t off = 0, total = 0;  // first task of this lane, tasks in all
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const unsigned m = __ballot_sync(FULL, (cnt >> b) & 1u);
        off += (uint32_t)__popc(m & lt) << b;
        total += (uint32_t)__popc(m) << b;
      }
      if (cnt > 0u) S.own[__popc(owners & lt)] = make_uint2(leaf_first(ref) - off, (uint32_t)lane | (off << 8));
      __syncwarp();
      int before = -1;  // owners whose first task lies before this group of 32
      for (uint32_t t0 = 0; t0 < total; t0 += 32) {
        const unsigned firsts = __reduce_or_sync(FULL, cnt > 0u && (off >> 5) == (t0 >> 5) ? 1u << (off & 31u) : 0u);
        const uint2 w = S.own[before + __popc(firsts & (0xffffffffu >> (31 - lane)))];
        before += __popc(firsts);
        const int o = (int)(w.y & 31u);
        const V3 qo{__shfl_sync(FULL, r.o.x, o), __shfl_sync(FULL, r.o.y, o), __shfl_sync(FULL, r.o.z, o)};
        const V3 qd{__shfl_sync(FULL, r.d.x, o), __shfl_sync(FULL, r.d.y, o), __shfl_sync(FULL, r.d.z, o)};
        const uint32_t t = t0 + (uint32_t)lane;
        if (t < total) {
          const Tri tr = load_tri(tris, w.x + t);
          float th = ray_tri(tr, qo, qd);
          if (th > 0.0f && th < max_t) {
            const float ndotd = vdot(tri_normal(tr), qd);
            if (ndotd > -1e-4f && ndotd < 1e-4f) th = INFINITY;  // grazing
            else if (!(ndotd > 0.0f)) th = -th;
          } else {
            th = INFINITY;
          }
          S.trid[(t - (w.y >> 8)) * kTriRow + o] = th;
        }
      }
      __syncwarp();
      if (cnt > 0u) {
        for (uint32_t k = 0; k < cnt; ++k) {
          const float t = S.trid[k * kTriRow + lane];
          if (t < INFINITY) {
            if (nh < kParityHits) S.hits[nh++][lane] = t;
            else if (nh < kParityCap) more_hits[nh++ - kParityHits] = t;
            else lost = true;
          }
        }
        ref = pop();
      }
      __syncwarp();
    }
    // (c) finished rays vote, new ones; without one the rest is passed by, which a
    // call of few rays waits for
    const bool done = live && ref == kNoItem;
    if (!__any_sync(FULL, done)) continue;
    bool vote = false;
    if (done && nh <= kParityHits) {
      // insertion sort by t
      for (int k = 1; k < nh; ++k) {
        const float t = S.hits[k][lane];
        int j = k;
        while (j > 0 && fabsf(S.hits[j - 1][lane]) > fabsf(t)) {
          S.hits[j][lane] = S.hits[j - 1][lane];
          --j;
        }
        S.hits[j][lane] = t;
      }
      vote = parity_vote(nh, coalesce, [&](int j, float& t, int& sg) {
        const float h = S.hits[j][lane];
        t = fabsf(h);
        sg = h < 0.f ? -1 : 1;
      });
    }
    for (unsigned m = __ballot_sync(FULL, done && nh > kParityHits); m; m &= m - 1u) {
      // the warp sorts one ray's hits: each goes to its rank
      const int o = __ffs(m) - 1, k = __shfl_sync(FULL, nh, o);
      if (lane == o)
        for (int j = kParityHits; j < k; ++j) S.trid[j] = more_hits[j - kParityHits];
      if (lane < kParityHits) S.trid[lane] = S.hits[lane][o];
      __syncwarp();
      for (int e = lane; e < k; e += 32) {
        const float t = S.trid[e];
        int rank = 0;
        for (int j = 0; j < k; ++j) {
          const float u = fabsf(S.trid[j]);
          rank += u < fabsf(t) || (u == fabsf(t) && j < e) ? 1 : 0;
        }
        S.sorted[rank] = t;
      }
      __syncwarp();
      if (lane == o)
        vote = parity_vote(k, coalesce, [&](int j, float& t, int& sg) {
          t = fabsf(S.sorted[j]);
          sg = S.sorted[j] < 0.f ? -1 : 1;
        });
      __syncwarp();
    }
    if (done) {
      if (vote) atomicAdd(&votes[i], 1);
      live = false;
    }
    const unsigned free_lanes = __ballot_sync(FULL, !live);
    if (!exhausted || pos < end) distribute(free_lanes);
  }
  if (lost) atomicExch(overflow, 1u);  // more hits or stack entries than a ray keeps
}

}  // namespace

}  // namespace a3d

using namespace a3d;

extern "C" size_t a3d_ray_workspace_bytes(int64_t num_rays) {
  Workspace ws(nullptr, 0);
  ws.take<uint32_t>(4);
  ws.take<uint32_t>(num_rays > 0 ? num_rays : 1);
  ws.take<int32_t>(num_rays > 0 ? num_rays : 1);
  ws.take<uint32_t>((int64_t)scan_workspace_elems(num_rays > 0 ? num_rays : 1) * 2);
  return ws.used + 256;
}

namespace {
// resident blocks of a persistent kernel, queried once per device
template <auto kKernel>
int blocks_per_sm(int* out) {
  static int cached[kMaxDevices] = {};
  int dev = 0;
  A3D_CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 0 && dev < kMaxDevices && cached[dev] > 0) {
    *out = cached[dev];
    return A3D_OK;
  }
  int b = 0;
  A3D_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kKernel, kRayThreads, 0));
  b = b < 1 ? 1 : b;
  if (dev >= 0 && dev < kMaxDevices) cached[dev] = b;
  *out = b;
  return A3D_OK;
}

// rays a warp takes at a time: 32 while that is under four pools a warp, at
// most kRayPool
int64_t ray_pool(int64_t rays, int64_t warps) {
  const int64_t pool = rays / (warps * 4) / 32 * 32;
  return pool < 32 ? 32 : (pool > kRayPool ? kRayPool : pool);
}

struct RayWs {
  uint32_t* status;  // [0] re-run count, [1] stack / buffer overflow, [2] pools taken
  uint32_t* rerun;
  int32_t* counts;
  int64_t* scan_tmp;
};
bool carve_ray(RayWs& w, void* p, size_t bytes, int64_t n) {
  Workspace ws(p, bytes);
  w.status = ws.take<uint32_t>(4);
  w.rerun = ws.take<uint32_t>(n > 0 ? n : 1);
  w.counts = ws.take<int32_t>(n > 0 ? n : 1);
  w.scan_tmp = ws.take<int64_t>((int64_t)scan_workspace_elems(n > 0 ? n : 1));
  return p && ws.ok();
}
}  // namespace

extern "C" int a3d_ray_nearest(const a3d_bvh_view* bvh, const float* rays_o, const float* rays_d, int64_t num_rays,
                               float max_t, const float* face_normals, uint8_t* hit, float* t, int32_t* face_ids,
                               float* hit_points, float* normals, float* uvw, void* workspace,
                               size_t workspace_bytes, a3d_stream_t stream_) {
  cudaStream_t s = (cudaStream_t)stream_;
  A3D_REQUIRE(bvh && bvh->nodes && bvh->tris, A3D_ERR_ARGUMENT, "ray_nearest: invalid bvh");
  A3D_REQUIRE(num_rays >= 0 && num_rays < (1ll << 32), A3D_ERR_ARGUMENT, "ray_nearest: bad number of rays");
  RayWs w;
  A3D_REQUIRE(carve_ray(w, workspace, workspace_bytes, num_rays), A3D_ERR_WORKSPACE, "ray_nearest: workspace");
  A3D_CUDA_TRY(cudaMemsetAsync(w.status, 0, 4 * sizeof(uint32_t), s));
  if (num_rays == 0) return A3D_OK;
  A3D_REQUIRE(rays_o && rays_d && hit && t && face_ids, A3D_ERR_ARGUMENT, "ray_nearest: null pointer");
  A3D_REQUIRE(normals == nullptr || face_normals != nullptr, A3D_ERR_ARGUMENT,
              "ray_nearest: normals need the face normals");
  const WideNode* nodes = (const WideNode*)bvh->nodes;
  const TriRec* tris = (const TriRec*)bvh->tris;
  const RayOut out{hit, t, face_ids, hit_points, normals, uvw};
  if (bvh->num_nodes <= kRayWholeNodes) {
    A3D_PDL(ray_whole_kernel, dim3((unsigned)ceil_div(num_rays, kRayThreads)), dim3(kRayThreads), 0, s, nodes,
            tris, face_normals, rays_o, rays_d, num_rays, max_t, out, w.status + 1);
    return A3D_OK;
  }
  int bps = 0;
  A3D_TRY(blocks_per_sm<ray_nearest_kernel>(&bps));
  const int64_t warps = (int64_t)num_sms() * bps * kRayWarps;
  const int64_t pool = ray_pool(num_rays, warps);
  const int64_t want = ceil_div(ceil_div(num_rays, pool), kRayWarps), cap = warps / kRayWarps;
  A3D_PDL(ray_nearest_kernel, dim3((unsigned)(want < cap ? want : cap)), dim3(kRayThreads), 0, s, nodes, tris, rays_o,
          rays_d, (uint32_t)num_rays, max_t, t, face_ids, w.rerun, w.status, w.status + 2, (uint32_t)pool);
  A3D_PDL(ray_nearest_rerun_kernel, dim3(num_sms() * 4), dim3(64), 0, s, nodes, tris, rays_o, rays_d, max_t, t,
          face_ids, w.rerun, w.status, w.status + 1);
  A3D_PDL(ray_finish_kernel, dim3((unsigned)ceil_div(num_rays, 256)), dim3(256), 0, s, tris, face_normals, rays_o,
          rays_d, num_rays, out);
  return A3D_OK;
}

extern "C" int a3d_ray_all_count(const a3d_bvh_view* bvh, const float* rays_o, const float* rays_d, int64_t num_rays,
                                 float max_t, int64_t* offsets_out, void* workspace, size_t workspace_bytes,
                                 a3d_stream_t stream_) {
  cudaStream_t s = (cudaStream_t)stream_;
  A3D_REQUIRE(bvh && bvh->nodes && bvh->tris, A3D_ERR_ARGUMENT, "ray_all: invalid bvh");
  A3D_REQUIRE(num_rays >= 0 && num_rays < (1ll << 32) && offsets_out, A3D_ERR_ARGUMENT, "ray_all: bad argument");
  RayWs w;
  A3D_REQUIRE(carve_ray(w, workspace, workspace_bytes, num_rays), A3D_ERR_WORKSPACE, "ray_all: workspace");
  A3D_CUDA_TRY(cudaMemsetAsync(w.status, 0, 4 * sizeof(uint32_t), s));
  if (num_rays == 0) return cudaMemsetAsync(offsets_out, 0, sizeof(int64_t), s) == cudaSuccess ? A3D_OK : A3D_ERR_CUDA;
  A3D_REQUIRE(rays_o && rays_d, A3D_ERR_ARGUMENT, "ray_all: null pointer");
  A3D_PDL(ray_all_count_kernel, dim3((unsigned)ceil_div(num_rays, 128)), dim3(128), 0, s, (const WideNode*)bvh->nodes,
          (const TriRec*)bvh->tris, rays_o, rays_d, num_rays, max_t, w.counts, w.status + 1);
  A3D_TRY((device_exclusive_scan<int32_t, int64_t>(w.counts, offsets_out, num_rays, w.scan_tmp,
                                                   offsets_out + num_rays, s)));
  return A3D_OK;
}

extern "C" int a3d_ray_all_collect(const a3d_bvh_view* bvh, const float* rays_o, const float* rays_d,
                                   int64_t num_rays, float max_t, const int64_t* offsets, int32_t* ray_idx,
                                   float* t, int32_t* face_ids, int32_t* sign, float* hit_points, float* uvw,
                                   a3d_stream_t stream_) {
  cudaStream_t s = (cudaStream_t)stream_;
  A3D_REQUIRE(bvh && bvh->nodes && bvh->tris, A3D_ERR_ARGUMENT, "ray_all: invalid bvh");
  A3D_REQUIRE(num_rays >= 0 && num_rays < (1ll << 32), A3D_ERR_ARGUMENT, "ray_all: bad number of rays");
  if (num_rays == 0) return A3D_OK;
  A3D_REQUIRE(rays_o && rays_d && offsets && ray_idx && t && face_ids && sign, A3D_ERR_ARGUMENT,
              "ray_all: null pointer");
  const AllOut out{ray_idx, t, face_ids, sign, hit_points, uvw};
  A3D_PDL(ray_all_collect_kernel, dim3((unsigned)ceil_div(num_rays, 128)), dim3(128), 0, s, (const WideNode*)bvh->nodes,
          (const TriRec*)bvh->tris, rays_o, rays_d, num_rays, max_t, offsets, out);
  return A3D_OK;
}

extern "C" int a3d_ray_parity_votes(const a3d_bvh_view* bvh, const float* points, int64_t num_points,
                                    const float* dirs, int32_t num_dirs, float max_t, float coalesce_t,
                                    int32_t* votes, void* workspace, size_t workspace_bytes, a3d_stream_t stream_) {
  cudaStream_t s = (cudaStream_t)stream_;
  A3D_REQUIRE(bvh && bvh->nodes && bvh->tris, A3D_ERR_ARGUMENT, "ray_parity: invalid bvh");
  A3D_REQUIRE(num_points >= 0 && num_dirs > 0 && num_dirs <= 1024, A3D_ERR_ARGUMENT, "ray_parity: bad argument");
  RayWs w;
  A3D_REQUIRE(carve_ray(w, workspace, workspace_bytes, 0), A3D_ERR_WORKSPACE, "ray_parity: workspace");
  A3D_CUDA_TRY(cudaMemsetAsync(w.status, 0, 4 * sizeof(uint32_t), s));
  if (num_points == 0) return A3D_OK;
  A3D_REQUIRE(points && dirs && votes, A3D_ERR_ARGUMENT, "ray_parity: null pointer");
  A3D_CUDA_TRY(cudaMemsetAsync(votes, 0, (size_t)num_points * sizeof(int32_t), s));
  int bps = 0;
  A3D_TRY(blocks_per_sm<ray_parity_kernel>(&bps));
  const int64_t rays = num_points * num_dirs, warps = (int64_t)num_sms() * bps * kRayWarps;
  const int64_t pool = ray_pool(rays, warps);
  const int64_t want = ceil_div(ceil_div(rays, pool), kRayWarps), cap = warps / kRayWarps;
  A3D_PDL(ray_parity_kernel, dim3((unsigned)(want < cap ? want : cap)), dim3(kRayThreads), 0, s,
          (const WideNode*)bvh->nodes, (const TriRec*)bvh->tris, points, num_points, dirs, num_dirs, max_t, coalesce_t,
          votes, w.status + 1, reinterpret_cast<unsigned long long*>(w.status + 2), pool);
  return A3D_OK;
}

extern "C" int a3d_ray_status(const void* workspace, uint32_t* status_out, a3d_stream_t stream) {
  A3D_REQUIRE(workspace && status_out, A3D_ERR_ARGUMENT, "ray_status: null pointer");
  A3D_CUDA_TRY(cudaMemcpyAsync(status_out, workspace, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                               (cudaStream_t)stream));
  A3D_CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
  return A3D_OK;
}
