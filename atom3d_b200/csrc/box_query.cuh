// Triangle/box SAT and the box query over the wide BVH, shared by the
// octree descent, MeshBVH.intersect_aabb's hit mask and its pair modes.
//
// SAT follows triangle_aabb_sat (atom3d/kernels/bvh_kernels.cu:285-353)
// operation by operation (box centre/half extents, 3 box axes, 9 edge cross
// axes, triangle plane, sat_eps = 1e-6).  Every multiply/add is an explicit
// round-to-nearest intrinsic so the compiler cannot contract it into an FMA:
// the result is then a pure function of IEEE single arithmetic and the CPU
// oracle (compiled with -ffp-contract=off) reproduces it bit for bit.
//
// The BVH only prunes: boxes are tested against child bounds grown by a
// margin that covers sat_eps and the rounding of the centre/half
// computation, so the set of triangles passing SAT does not depend on the
// tree.
#pragma once

#include <math.h>

#include "a3d_common.cuh"
#include "bvh_layout.cuh"

namespace a3d {

constexpr int kSatThreads = 128;
constexpr int kSatDepth = 48;
constexpr int kSatDeepDepth = 512;

__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsb(float a, float b) { return __fsub_rn(a, b); }

__device__ __forceinline__ float dot3r(float ax, float ay, float az, float bx, float by, float bz) {
  return fa(fa(fm(ax, bx), fm(ay, by)), fm(az, bz));
}

// The edge and plane axes in full, for operands that are not all finite.
static __device__ __noinline__ bool sat_general(float v0x, float v0y, float v0z, float v1x, float v1y, float v1z, float v2x,
                                         float v2y, float v2z, float hx, float hy, float hz) {
  const float eps = 1e-6f;
  const float e[3][3] = {{fsb(v1x, v0x), fsb(v1y, v0y), fsb(v1z, v0z)},
                         {fsb(v2x, v1x), fsb(v2y, v1y), fsb(v2z, v1z)},
                         {fsb(v0x, v2x), fsb(v0y, v2y), fsb(v0z, v2z)}};
  for (int k = 0; k < 3; ++k) {
    const float ex = e[k][0], ey = e[k][1], ez = e[k][2];
    for (int ax = 0; ax < 3; ++ax) {
      float a0, a1, a2;
      if (ax == 0) { a0 = 0.f; a1 = ez; a2 = -ey; }
      else if (ax == 1) { a0 = -ez; a1 = 0.f; a2 = ex; }
      else { a0 = ey; a1 = -ex; a2 = 0.f; }
      const float p0 = dot3r(v0x, v0y, v0z, a0, a1, a2);
      const float p1 = dot3r(v1x, v1y, v1z, a0, a1, a2);
      const float p2 = dot3r(v2x, v2y, v2z, a0, a1, a2);
      const float mnp = fminf(fminf(p0, p1), p2), mxp = fmaxf(fmaxf(p0, p1), p2);
      const float rad = fa(fa(fa(fm(hx, fabsf(a0)), fm(hy, fabsf(a1))), fm(hz, fabsf(a2))), eps);
      if (mnp > rad || mxp < -rad) return false;
    }
  }
  const float wx = fsb(v2x, v0x), wy = fsb(v2y, v0y), wz = fsb(v2z, v0z);
  const float nx = fsb(fm(e[0][1], wz), fm(e[0][2], wy));
  const float ny = fsb(fm(e[0][2], wx), fm(e[0][0], wz));
  const float nz = fsb(fm(e[0][0], wy), fm(e[0][1], wx));
  const float d = -dot3r(nx, ny, nz, v0x, v0y, v0z);
  const float r = fa(fa(fa(fm(hx, fabsf(nx)), fm(hy, fabsf(ny))), fm(hz, fabsf(nz))), eps);
  return !(fabsf(d) > r);
}

// one edge axis: the projections of the two coordinates that its zero
// component leaves, against the radius
__device__ __forceinline__ bool sat_axis_apart(float u0, float w0, float u1, float w1, float u2, float w2, float au,
                                               float aw, float hu, float hw) {
  const float p0 = fa(fm(u0, au), fm(w0, aw)), p1 = fa(fm(u1, au), fm(w1, aw)), p2 = fa(fm(u2, au), fm(w2, aw));
  const float rad = fa(fa(fm(hu, fabsf(au)), fm(hw, fabsf(aw))), 1e-6f);
  return fminf(fminf(p0, p1), p2) > rad || fmaxf(fmaxf(p0, p1), p2) < -rad;
}

// Triangle a, b, c against the box of centre (cx, cy, cz) and half extents
// (hx, hy, hz).  The decision is an AND of 13 comparisons without side
// effects, so it does not depend on their order: the plane, which rejects most
// triangles whose own box meets the query's, comes before the nine edge axes.
// Each edge axis has a zero component; with finite operands its products add
// +-0, which changes no comparison, and are left out (a non-finite operand,
// whose product with 0 is NaN, takes sat_general).
__device__ __forceinline__ bool sat_half(const float4& a, const float4& b, const float4& c, float cx, float cy,
                                         float cz, float hx, float hy, float hz) {
  const float eps = 1e-6f;
  const float v0x = fsb(a.x, cx), v0y = fsb(a.y, cy), v0z = fsb(a.z, cz);
  const float v1x = fsb(b.x, cx), v1y = fsb(b.y, cy), v1z = fsb(b.z, cz);
  const float v2x = fsb(c.x, cx), v2y = fsb(c.y, cy), v2z = fsb(c.z, cz);
  if (fminf(fminf(v0x, v1x), v2x) > fa(hx, eps) || fmaxf(fmaxf(v0x, v1x), v2x) < fsb(-hx, eps) ||
      fminf(fminf(v0y, v1y), v2y) > fa(hy, eps) || fmaxf(fmaxf(v0y, v1y), v2y) < fsb(-hy, eps) ||
      fminf(fminf(v0z, v1z), v2z) > fa(hz, eps) || fmaxf(fmaxf(v0z, v1z), v2z) < fsb(-hz, eps))
    return false;
  // 0, or NaN with an operand that is not finite or a sum that overflows, which
  // the general form decides the same (short chains: a walk waits for it)
  const float z = (((v0x + v0y) + (v0z + v1x)) + ((v1y + v1z) + (v2x + v2y)) + ((v2z + hx) + (hy + hz))) * 0.f;
  if (!(z == 0.f)) return sat_general(v0x, v0y, v0z, v1x, v1y, v1z, v2x, v2y, v2z, hx, hy, hz);
  const float e0x = fsb(v1x, v0x), e0y = fsb(v1y, v0y), e0z = fsb(v1z, v0z);
  {  // plane: normal = cross(e0, v2 - v0)
    const float wx = fsb(v2x, v0x), wy = fsb(v2y, v0y), wz = fsb(v2z, v0z);
    const float nx = fsb(fm(e0y, wz), fm(e0z, wy));
    const float ny = fsb(fm(e0z, wx), fm(e0x, wz));
    const float nz = fsb(fm(e0x, wy), fm(e0y, wx));
    const float d = -dot3r(nx, ny, nz, v0x, v0y, v0z);
    const float r = fa(fa(fa(fm(hx, fabsf(nx)), fm(hy, fabsf(ny))), fm(hz, fabsf(nz))), eps);
    if (fabsf(d) > r) return false;
  }
  const float e[3][3] = {{e0x, e0y, e0z},
                         {fsb(v2x, v1x), fsb(v2y, v1y), fsb(v2z, v1z)},
                         {fsb(v0x, v2x), fsb(v0y, v2y), fsb(v0z, v2z)}};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float ex = e[k][0], ey = e[k][1], ez = e[k][2];
    if (sat_axis_apart(v0y, v0z, v1y, v1z, v2y, v2z, ez, -ey, hy, hz) ||
        sat_axis_apart(v0x, v0z, v1x, v1z, v2x, v2z, -ez, ex, hx, hz) ||
        sat_axis_apart(v0x, v0y, v1x, v1y, v2x, v2y, ey, -ex, hx, hy))
      return false;
  }
  return true;
}

// box centre and half extents as the SAT rounds them
__device__ __forceinline__ float box_centre(float mn, float mx) { return fm(fa(mn, mx), 0.5f); }
__device__ __forceinline__ float box_half(float mn, float mx) { return fm(fsb(mx, mn), 0.5f); }

__device__ __forceinline__ bool sat_test(const TriRec& t, float mnx, float mny, float mnz, float mxx, float mxy, float mxz) {
  return sat_half(t.a, t.b, t.c, box_centre(mnx, mxx), box_centre(mny, mxy), box_centre(mnz, mxz), box_half(mnx, mxx),
                  box_half(mny, mxy), box_half(mnz, mxz));
}

struct ShStack {
  uint32_t* base;
  int sp;
  static constexpr int kDepth = kSatDepth;
  __device__ __forceinline__ void push(uint32_t r) { base[sp++ * kSatThreads] = r; }
  __device__ __forceinline__ uint32_t pop() { return base[--sp * kSatThreads]; }
};
struct LcStack {
  uint32_t s[kSatDeepDepth];
  int sp;
  static constexpr int kDepth = kSatDeepDepth;
  __device__ __forceinline__ void push(uint32_t r) { s[sp++] = r; }
  __device__ __forceinline__ uint32_t pop() { return s[--sp]; }
};

// margin of the pruning box, covering sat_eps and rounding
__device__ __forceinline__ float box_margin(float mnx, float mny, float mnz, float mxx, float mxy, float mxz) {
  const float mag = fmaxf(fmaxf(fmaxf(fabsf(mnx), fabsf(mxx)), fmaxf(fabsf(mny), fabsf(mxy))),
                          fmaxf(fabsf(mnz), fabsf(mxz)));
  return 4e-6f + 4e-7f * mag;
}

// Visits every leaf triangle of the tree whose box may meet the query box;
// visit(const TriRec& t, uint32_t slot) returns true to stop.  Returns 0 =
// finished, 1 = stopped by visit, 2 = stack overflow.  Children are pushed
// last-first, so leaves are visited in a fixed (tree) order.
template <typename Stack, typename Visit>
__device__ __forceinline__ int box_traverse(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                                            float mnx, float mny, float mnz, float mxx, float mxy, float mxz,
                                            Stack& st, Visit&& visit) {
  const float g = box_margin(mnx, mny, mnz, mxx, mxy, mxz);
  const float lx = mnx - g, ly = mny - g, lz = mnz - g, ux = mxx + g, uy = mxy + g, uz = mxz + g;
  uint32_t ref = 0;
  for (;;) {
    if (!ref_is_leaf(ref)) {
      const int4* np = reinterpret_cast<const int4*>(nodes + ref);
      const int4 w0 = __ldg(np), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3);
      const float ox = __int_as_float(w0.x), oy = __int_as_float(w0.y), oz = __int_as_float(w0.z);
      const uint32_t meta = (uint32_t)w0.w;
      const float sx = __uint_as_float((meta & 0xffu) << 23);
      const float sy = __uint_as_float(((meta >> 8) & 0xffu) << 23);
      const float sz = __uint_as_float(((meta >> 16) & 0xffu) << 23);
      const int nch = (int)(meta >> 24);
      const uint32_t r[4] = {(uint32_t)w2.z, (uint32_t)w2.w, (uint32_t)w3.x, (uint32_t)w3.y};
      for (int c = nch - 1; c >= 0; --c) {
        const float clx = dequant((uint32_t)w1.x, c, sx, ox);
        const float cly = dequant((uint32_t)w1.y, c, sy, oy);
        const float clz = dequant((uint32_t)w1.z, c, sz, oz);
        const float chx = dequant((uint32_t)w1.w, c, sx, ox);
        const float chy = dequant((uint32_t)w2.x, c, sy, oy);
        const float chz = dequant((uint32_t)w2.y, c, sz, oz);
        const bool ov = clx <= ux && chx >= lx && cly <= uy && chy >= ly && clz <= uz && chz >= lz;
        if (ov) {
          if (st.sp >= Stack::kDepth) return 2;
          st.push(r[c]);
        }
      }
    } else {
      const uint32_t f0 = leaf_first(ref), cnt = leaf_count(ref);
      for (uint32_t i = 0; i < cnt; ++i) {
        const float4* p = reinterpret_cast<const float4*>(tris + f0 + i);
        TriRec t;
        t.a = __ldg(p); t.b = __ldg(p + 1); t.c = __ldg(p + 2); t.r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (visit(t, f0 + i)) return 1;
      }
    }
    if (st.sp == 0) return 0;
    ref = st.pop();
  }
}


// any-hit SAT query; returns 0 = miss, 1 = hit, 2 = stack overflow
template <typename Stack>
__device__ int box_any_hit(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris, float mnx, float mny,
                           float mnz, float mxx, float mxy, float mxz, Stack& st) {
  return box_traverse(nodes, tris, mnx, mny, mnz, mxx, mxy, mxz, st, [&](const TriRec& t, uint32_t) {
    return sat_test(t, mnx, mny, mnz, mxx, mxy, mxz);
  });
}

// ---- the walk of a warp ---------------------------------------------------------
constexpr int kBoxThreads = 128;
constexpr int kBoxWarps = kBoxThreads / 32;
// stack entries of a box in shared memory; the rest, to kSatDeepDepth, go to local
// memory (with a second walk by one lane for the boxes that need them, 100 boxes
// of 195,858 pairs each among 300,000 triangles of all sizes took 1.18 s, now
// 0.23; 0.85 with a thread a box)
constexpr int kLaneDepth = 32;
constexpr int kBoxBlocks = 7;  // resident blocks an SM
constexpr int kBoxNodeLanes = 4;  // boxes at a node below which a warp turns to its leaves
constexpr int kBoxRefill = 16;  // free lanes that are given new boxes together
constexpr int kBoxItems = 256;    // most boxes a warp takes
constexpr uint32_t kNoRef = 0xffffffffu;    // no node, leaf or triangle: no reference has this value

struct BoxSmem {
  uint32_t stack[kLaneDepth][32];
  float box[6][32];       // centre and half extents of each lane's box
  uint8_t task[32 * kMaxLeafTris];  // a leaf step's tests: lane | position in its leaf << 5
};

// Boxes a warp takes: all warps get some while there are few, down to one each,
// since a warp's time is that of all its boxes' steps (1,000 boxes of some 150
// pairs each, 1,310,720 triangles: count and write pass 377 + 655 us at 32 boxes a
// warp, 253 + 301 at one; a thread a box 448 + 488).
__host__ __device__ inline int64_t box_items(int64_t n, int64_t warps) {
  const int64_t per = ceil_div(n, warps);
  return per <= 32 ? (per < 1 ? 1 : per) : per > kBoxItems ? kBoxItems : ceil_div(per, 32) * 32;
}

// A query Q of the walk (its members are the state of the lane's box):
//   begin(i, mn, mx)   the box of item i
//   leaf(mask, first)  bit k: triangle first + k passed SAT
//   done(overflow)     the walk is over, or outgrew its stack

// pruning box of a lane
struct PruneBox {
  float lx, ly, lz, ux, uy, uz;
};
__device__ __forceinline__ PruneBox set_box(BoxSmem& S, const float* mn, const float* mx) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    S.box[a][lane] = box_centre(mn[a], mx[a]);
    S.box[3 + a][lane] = box_half(mn[a], mx[a]);
  }
  const float g = box_margin(mn[0], mn[1], mn[2], mx[0], mx[1], mx[2]);
  return PruneBox{mn[0] - g, mn[1] - g, mn[2] - g, mx[0] + g, mx[1] + g, mx[2] + g};
}

// which children of a node meet the box; their references
__device__ __forceinline__ void child_overlap(const WideNode* __restrict__ nodes, uint32_t ref, const PruneBox& p,
                                              bool ov[4], uint32_t r[4]) {
  int4 w0, w1, w2, w3;
  ldg256(nodes + ref, w0, w1);
  ldg256(reinterpret_cast<const char*>(nodes + ref) + 32, w2, w3);
  const float ox = __int_as_float(w0.x), oy = __int_as_float(w0.y), oz = __int_as_float(w0.z);
  const uint32_t meta = (uint32_t)w0.w;
  const float sx = __uint_as_float((meta & 0xffu) << 23);
  const float sy = __uint_as_float(((meta >> 8) & 0xffu) << 23);
  const float sz = __uint_as_float(((meta >> 16) & 0xffu) << 23);
  const int nch = (int)(meta >> 24);
  r[0] = (uint32_t)w2.z; r[1] = (uint32_t)w2.w; r[2] = (uint32_t)w3.x; r[3] = (uint32_t)w3.y;
#pragma unroll
  for (int c = 0; c < 4; ++c)
    ov[c] = c < nch && dequant((uint32_t)w1.x, c, sx, ox) <= p.ux && dequant((uint32_t)w1.w, c, sx, ox) >= p.lx &&
            dequant((uint32_t)w1.y, c, sy, oy) <= p.uy && dequant((uint32_t)w2.x, c, sy, oy) >= p.ly &&
            dequant((uint32_t)w1.z, c, sz, oz) <= p.uz && dequant((uint32_t)w2.y, c, sz, oz) >= p.lz;
}

// One leaf step: the cnt triangles (0: none) from first on of every lane's box.
// Each lane compares its triangles' own boxes with its box (about a third of
// them meet it); the rest of the test, five times as long, is spread evenly
// over the lanes.  Where the triangles of all lanes make one round of tests, or
// three quarters of the last step's passed (dense), the comparison costs more
// than it saves and is left out (1,000 boxes of 342 pairs, 1,310,720 triangles:
// 994 -> 772 us a call; 5,000 boxes that each hold a quarter of 100,000
// triangles 74.9 -> 57.2 ms, 101 with a thread a box).  Returns the mask of the
// lane's triangles that pass SAT.
__device__ __forceinline__ uint32_t leaf_step(const TriRec* __restrict__ tris, uint32_t cnt, uint32_t first,
                                              const PruneBox& pb, BoxSmem& S, bool& dense) {
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t tris_here = __reduce_add_sync(FULL, cnt);
  const bool all = dense || tris_here <= 32u;
  uint32_t near = all ? (1u << cnt) - 1u : 0u;
  const float4* p = reinterpret_cast<const float4*>(tris + first);
  for (uint32_t k = all ? cnt : 0u; k < cnt; ++k, p += 4) {
    const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
    if (!(fminf(fminf(a.x, b.x), c.x) > pb.ux || fmaxf(fmaxf(a.x, b.x), c.x) < pb.lx ||
          fminf(fminf(a.y, b.y), c.y) > pb.uy || fmaxf(fmaxf(a.y, b.y), c.y) < pb.ly ||
          fminf(fminf(a.z, b.z), c.z) > pb.uz || fmaxf(fmaxf(a.z, b.z), c.z) < pb.lz))
      near |= 1u << k;
  }
  const uint32_t num = (uint32_t)__popc(near);
  uint32_t off = 0, total = 0;  // first test of this lane, tests in all
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const unsigned m = __ballot_sync(FULL, (num >> b) & 1u);
    off += (uint32_t)__popc(m & lt) << b;
    total += (uint32_t)__popc(m) << b;
  }
  {
    uint32_t j = off;
    for (uint32_t m = near; m; m &= m - 1u) S.task[j++] = (uint8_t)(lane | (__ffs((int)m) - 1) << 5);
  }
  __syncwarp();
  uint32_t hits = 0;  // bit j: the j-th near triangle passes
  uint32_t passed = 0;
  for (uint32_t t0 = 0; t0 < total; t0 += 32) {
    const uint32_t t = t0 + (uint32_t)lane;
    const uint32_t w = t < total ? S.task[t] : 0u;
    const int o = (int)(w & 31u);
    const uint32_t slot = __shfl_sync(FULL, first, o) + (w >> 5);
    bool pass = false;
    if (t < total) {
      const float4* q = reinterpret_cast<const float4*>(tris + slot);
      const float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
      pass = sat_half(a, b, c, S.box[0][o], S.box[1][o], S.box[2][o], S.box[3][o], S.box[4][o], S.box[5][o]);
    }
    const unsigned r = __ballot_sync(FULL, pass);
    passed += (uint32_t)__popc(r);
    if (off + num > t0 && off < t0 + 32u) hits |= off >= t0 ? r >> (off - t0) : r << (t0 - off);
  }
  __syncwarp();
  dense = 4u * passed >= 3u * tris_here;
  uint32_t mask = 0;
  for (uint32_t m = near; m; m &= m - 1u, hits >>= 1)
    if (hits & 1u) mask |= m & (0u - m);
  return mask;
}

// The boxes [pos, end) of a warp, one box a lane; kBoxRefill lanes that are done
// get new ones together.  The warp alternates node steps, while at least
// kBoxNodeLanes of its boxes are at an inner node, with one leaf step.  Each box
// visits the tree in box_traverse's order.
// Bound by its instructions, 17 of 32 lanes active (box_traverse: 8): a box of
// 3 pairs visits 10 nodes and 2.4 leaves of 13 triangles.  Counting the pairs
// of 933,270 voxels with 327,680 triangles: 438 -> 351 us.  A walk shared by
// eight neighbouring boxes took 460 us, the triangles spread over the lanes
// before their boxes are compared 413; 20 / 8 / 1 node lanes 413 / 356 / 362 us.
// Any-hit queries stay with box_traverse, where the walk ends at the first hit:
// the octree's voxels (0.70 ms) took 0.80 ms this way.
template <typename Query>
__device__ __forceinline__ void box_walk(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                                          int64_t pos, int64_t end, BoxSmem& S, Query& q) {
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  const unsigned lt = (1u << lane) - 1u;
  bool live = false, over = false, dense = false;
  int sp = 0;
  uint32_t ref = kNoRef;
  PruneBox pb{};
  uint32_t more[kSatDeepDepth - kLaneDepth];
  const uint32_t* deep = more;
  auto pop = [&]() -> uint32_t {
    if (sp == 0) return kNoRef;
    --sp;
    return sp < kLaneDepth ? S.stack[sp][lane] : deep[sp - kLaneDepth];
  };
  for (;;) {
    // (a) new boxes
    const unsigned want = __ballot_sync(FULL, !live);
    if (__popc(want) >= kBoxRefill && pos < end) {
      const int64_t i = pos + __popc(want & lt);
      if (!live && i < end) {
        float mn[3], mx[3];
        q.begin(i, mn, mx);
        pb = set_box(S, mn, mx);
        sp = 0;
        ref = 0u;
        live = true;
        over = false;
      }
      pos = pos + __popc(want) < end ? pos + __popc(want) : end;
      __syncwarp();
    }
    if (!__any_sync(FULL, live)) break;
    // (b) node steps
    for (;;) {
      const unsigned at_node = __ballot_sync(FULL, (int)ref >= 0);
      if (__popc(at_node) < kBoxNodeLanes && (at_node == 0u || __any_sync(FULL, live && (int)ref < 0))) break;
      if ((int)ref >= 0) {
        bool ov[4];
        uint32_t r[4];
        child_overlap(nodes, ref, pb, ov, r);
        uint32_t next = kNoRef;
#pragma unroll
        for (int c = 3; c >= 0; --c)
          if (ov[c]) {
            if (next != kNoRef) {
              if (sp < kLaneDepth) S.stack[sp++][lane] = next;
              else if (sp < kSatDeepDepth) more[sp++ - kLaneDepth] = next;
              else over = true;
            }
            next = r[c];
          }
        if (next == kNoRef) next = pop();
        ref = over ? kNoRef : next;
      }
    }
    // (c) leaf step
    const uint32_t cnt = live && (int)ref < 0 && ref != kNoRef ? leaf_count(ref) : 0u;
    if (__any_sync(FULL, cnt > 0u)) {
      const uint32_t mask = leaf_step(tris, cnt, leaf_first(ref), pb, S, dense);
      if (cnt > 0u) {
        if (mask) q.leaf(mask, leaf_first(ref));
        ref = pop();
      }
    }
    // (d) finished boxes
    if (live && ref == kNoRef) {
      q.done(over);
      live = false;
    }
  }
}

// all warps of the grid share the n items
template <typename Query>
__device__ __forceinline__ void box_walk_all(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                                              int64_t n, BoxSmem& S, Query& q) {
  const int64_t warps = (int64_t)gridDim.x * kBoxWarps, per = box_items(n, warps);
  for (int64_t pos = ((int64_t)blockIdx.x * kBoxWarps + (threadIdx.x >> 5)) * per; pos < n; pos += warps * per)
    box_walk(nodes, tris, pos, pos + per < n ? pos + per : n, S, q);
}
// blocks of box_walk_all over at most n items
inline int64_t box_blocks(int64_t n, int sms) {
  const int64_t want = ceil_div(n, kBoxWarps), cap = (int64_t)sms * kBoxBlocks;
  return want < cap ? want : cap;
}

}  // namespace a3d
