// Morton keys, triangle/box SAT any-hit queries and the coarse-to-fine
// octree descent.  A box "hits" when some triangle passes SAT (the test and
// the tree walk are in box_query.cuh).
#include <math.h>

#include "box_query.cuh"
#include "primitives.cuh"

namespace a3d {

namespace {

// ---- explicit boxes (MeshBVH.intersect_aabb mode 0) -----------------------
__global__ void __launch_bounds__(kSatThreads)
    aabb_hit_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                    const float* __restrict__ bmin, const float* __restrict__ bmax, int64_t n,
                    uint8_t* __restrict__ hit, uint32_t* __restrict__ spill, uint32_t* __restrict__ nspill) {
  pdl_wait();
  __shared__ uint32_t s_stack[kSatDepth * kSatThreads];
  const int64_t i = (int64_t)blockIdx.x * kSatThreads + threadIdx.x;
  if (i >= n) return;
  ShStack st{s_stack + threadIdx.x, 0};
  const int r = box_any_hit(nodes, tris, bmin[3 * i], bmin[3 * i + 1], bmin[3 * i + 2], bmax[3 * i], bmax[3 * i + 1],
                            bmax[3 * i + 2], st);
  if (r == 2) {
    spill[atomicAdd(nspill, 1u)] = (uint32_t)i;
  } else {
    hit[i] = (uint8_t)r;
  }
}

__global__ void aabb_hit_spill_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                                      const float* __restrict__ bmin, const float* __restrict__ bmax,
                                      uint8_t* __restrict__ hit, const uint32_t* __restrict__ spill,
                                      const uint32_t* __restrict__ nspill, int* __restrict__ overflow) {
  pdl_wait();
  const uint32_t m = *nspill;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = spill[t];
    LcStack st;
    st.sp = 0;
    const int r = box_any_hit(nodes, tris, bmin[3 * i], bmin[3 * i + 1], bmin[3 * i + 2], bmax[3 * i],
                              bmax[3 * i + 1], bmax[3 * i + 2], st);
    if (r == 2) atomicExch(overflow, 1);
    hit[i] = r == 1 ? 1 : 0;
  }
}

// ---- octree levels ----------------------------------------------------------
struct LevelGeom {
  float lo[3];
  float cell[3];
};

__device__ __forceinline__ void cube_box(int x, int y, int z, const LevelGeom& g, float* mn, float* mx) {
  // aabb_min = float(ijk) * cell + lo ; aabb_max = aabb_min + cell  (two roundings, no FMA)
  const int ijk[3] = {x, y, z};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    mn[a] = fa(fm((float)ijk[a], g.cell[a]), g.lo[a]);
    mx[a] = fa(mn[a], g.cell[a]);
  }
}

// What a level knows about a hit voxel, in one word for its children: the
// place of its triangle list in the level's arena (below 2^31), or kHintBit and
// the triangle that hit it, or kNoHint.
constexpr uint32_t kNoHint = 0xffffffffu;
constexpr uint32_t kHintBit = 0x80000000u;
constexpr int kListMax = 32;  // triangles of a list
constexpr int64_t kListFull = 1 << 14;  // candidates that fill the chip

// candidate k of this level: either cube k of the full min_level grid
// (meshgrid 'ij': x slowest, z fastest) or child (k & 7) of parent k >> 3
__device__ __forceinline__ void candidate_ijk(int64_t k, bool first_level, int res, const int32_t* parents, int& x,
                                              int& y, int& z) {
  if (first_level) {
    x = (int)(k / ((int64_t)res * res));
    y = (int)((k / res) % res);
    z = (int)(k % res);
  } else {
    const int64_t p = k >> 3;
    const int c = (int)(k & 7);
    x = 2 * parents[3 * p] + (c & 1);
    y = 2 * parents[3 * p + 1] + ((c >> 1) & 1);
    z = 2 * parents[3 * p + 2] + ((c >> 2) & 1);
  }
}

// A candidate's hit decision: the triangle that hit its parent first (most
// children of a hit voxel meet the same triangle, which is several voxels
// wide at the finest levels), else an any-hit walk from the root.  The SAT
// predicate does not depend on the tree (the walk's pruning box is grown to
// cover sat_eps and rounding), so a hint that hits gives the decision the
// walk would give.  The hitting triangle's slot goes to the candidate's own
// children.
template <typename Stack>
__device__ __forceinline__ int candidate_hit(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                                             const float* mn, const float* mx, uint32_t hint, Stack& st,
                                             uint32_t& hit_slot) {
  if (hint != kNoHint) {
    const uint32_t slot = hint & ~kHintBit;
    const float4* p = reinterpret_cast<const float4*>(tris + slot);
    TriRec t;
    t.a = __ldg(p); t.b = __ldg(p + 1); t.c = __ldg(p + 2); t.r = make_float4(0.f, 0.f, 0.f, 0.f);
    if (sat_test(t, mn[0], mn[1], mn[2], mx[0], mx[1], mx[2])) {
      hit_slot = hint;
      return 1;
    }
  }
  return box_traverse(nodes, tris, mn[0], mn[1], mn[2], mx[0], mx[1], mx[2], st, [&](const TriRec& t, uint32_t slot) {
    if (!sat_test(t, mn[0], mn[1], mn[2], mx[0], mx[1], mx[2])) return false;
    hit_slot = slot | kHintBit;
    return true;
  });
}

struct Level {
  int64_t ncand;
  bool first_level;
  int res;
  const int32_t* parents;
  const uint32_t* parent_hint;
  LevelGeom g;
  uint32_t* flags;
  uint8_t* hit;
  uint32_t* ctri;
  uint32_t* spill;
  uint32_t* nspill;
  // triangle lists (the list kernels): the parents' arena, this level's, its
  // size in words and the words taken; margin of a list's box
  const uint32_t* parent_lists;
  uint32_t* lists;
  uint32_t list_cap;
  uint32_t* list_used;
  float margin;
};

__device__ __forceinline__ void put_decision(const Level& lv, int64_t k, int status, uint32_t info) {
  const uint32_t h = status == 1 ? 1u : 0u;
  lv.flags[k] = h;
  lv.hit[k] = (uint8_t)h;
  lv.ctri[k] = info;
  if (status == 2) lv.spill[atomicAdd(lv.nspill, 1u)] = (uint32_t)k;
}

__global__ void __launch_bounds__(kSatThreads)
    octree_level_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris, Level lv) {
  pdl_wait();
  __shared__ uint32_t s_stack[kSatDepth * kSatThreads];
  const int64_t k = (int64_t)blockIdx.x * kSatThreads + threadIdx.x;
  if (k >= lv.ncand) return;
  int x, y, z;
  candidate_ijk(k, lv.first_level, lv.res, lv.parents, x, y, z);
  float mn[3], mx[3];
  cube_box(x, y, z, lv.g, mn, mx);
  ShStack st{s_stack + threadIdx.x, 0};
  uint32_t info = kNoHint;
  const uint32_t hint = lv.parent_hint ? lv.parent_hint[k >> 3] : kNoHint;
  const int r = candidate_hit(nodes, tris, mn, mx, hint, st, info);
  put_decision(lv, k, r, info);
}

// ---- triangle lists ---------------------------------------------------------
// Once a voxel meets few triangles, walking the tree for each of its children,
// grandchildren and so on finds the same ones again and again.  One level
// collects each hit voxel's triangles in a walk, and the levels below test only
// their parent's list, and pass on what of it meets their own box.  A list holds
// every triangle whose own box meets the voxel's, grown by lv.margin: that covers
// sat_eps, the rounding of the test and of the boxes of all levels below, so a
// triangle that passes the SAT of any descendant is in it, and testing the list
// gives the decision of the walk.  A voxel with more than kListMax triangles (or
// a non-finite one), or whose list finds no room, has none; its children walk.
// Bound by instructions.  327,680 triangles: the finest level of a 512^3 grid
// (1.73M candidates), whose walks ran at 9 of 32 lanes, takes 132 instead of
// 399 us, the one above 73 instead of 125, the collecting one 127 instead of 57;
// the descent to 1024^3 0.9 instead of 2.04 ms.
struct GrownBox {
  float lx, ly, lz, ux, uy, uz;
};
__device__ __forceinline__ GrownBox grown(const float* mn, const float* mx, float g) {
  return GrownBox{mn[0] - g, mn[1] - g, mn[2] - g, mx[0] + g, mx[1] + g, mx[2] + g};
}
__device__ __forceinline__ bool meets(const float4& a, const float4& b, const float4& c, const GrownBox& q) {
  return !(fminf(fminf(a.x, b.x), c.x) > q.ux || fmaxf(fmaxf(a.x, b.x), c.x) < q.lx ||
           fminf(fminf(a.y, b.y), c.y) > q.uy || fmaxf(fmaxf(a.y, b.y), c.y) < q.ly ||
           fminf(fminf(a.z, b.z), c.z) > q.uz || fmaxf(fmaxf(a.z, b.z), c.z) < q.lz);
}

// Room for n words (0: none) of every lane; returns the lane's place, or
// kNoHint when the arena is full.  All lanes of the warp call it.
__device__ __forceinline__ uint32_t take_words(const Level& lv, uint32_t n) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  uint32_t incl = n;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t u = __shfl_up_sync(FULL, incl, d);
    if (lane >= d) incl += u;
  }
  const uint32_t total = __shfl_sync(FULL, incl, 31);
  uint32_t base = 0;
  if (lane == 0 && total) {
    base = lv.list_cap;  // full already: the count must not wrap
    if (*(volatile uint32_t*)lv.list_used < lv.list_cap) base = atomicAdd(lv.list_used, total);
  }
  base = __shfl_sync(FULL, base, 0);
  return base + total <= lv.list_cap && base < lv.list_cap ? base + incl - n : kNoHint;
}

// The level that collects: walks from the root.
__global__ void __launch_bounds__(kSatThreads)
    octree_collect_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris, Level lv) {
  pdl_wait();
  __shared__ uint32_t s_stack[kSatDepth * kSatThreads];
  const int64_t k = (int64_t)blockIdx.x * kSatThreads + threadIdx.x;
  uint32_t slots[kListMax];
  uint32_t num = 0, info = kNoHint;
  int r = 0;
  if (k < lv.ncand) {
    int x, y, z;
    candidate_ijk(k, lv.first_level, lv.res, lv.parents, x, y, z);
    float mn[3], mx[3];
    cube_box(x, y, z, lv.g, mn, mx);
    const GrownBox q = grown(mn, mx, lv.margin);
    ShStack st{s_stack + threadIdx.x, 0};
    r = box_traverse(nodes, tris, q.lx, q.ly, q.lz, q.ux, q.uy, q.uz, st, [&](const TriRec& t, uint32_t slot) {
      if (!meets(t.a, t.b, t.c, q)) return false;
      const float zero = (t.a.x + t.a.y + t.a.z + t.b.x + t.b.y + t.b.z + t.c.x + t.c.y + t.c.z) * 0.0f;
      if (num < (uint32_t)kListMax && zero == 0.0f) slots[num++] = slot;
      else num = kListMax + 1;
      if (info == kNoHint && sat_test(t, mn[0], mn[1], mn[2], mx[0], mx[1], mx[2])) info = slot | kHintBit;
      return info != kNoHint && num > (uint32_t)kListMax;
    });
    if (r != 2) r = info != kNoHint;
  }
  const bool list = r == 1 && num <= (uint32_t)kListMax;
  const uint32_t place = take_words(lv, list ? num + 1 : 0u);
  if (list && place != kNoHint) {
    lv.lists[place] = num;
    for (uint32_t j = 0; j < num; ++j) lv.lists[place + 1 + j] = slots[j];
    info = place;
  }
  if (k < lv.ncand) put_decision(lv, k, r, info);
}

// The levels below: eight lanes test the eight children of one parent.
template <bool kBuild>
__global__ void __launch_bounds__(kSatThreads)
    octree_list_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris, Level lv) {
  pdl_wait();
  __shared__ uint32_t s_stack[kSatDepth * kSatThreads];
  const int64_t k = (int64_t)blockIdx.x * kSatThreads + threadIdx.x;
  const uint32_t parent = k < lv.ncand ? lv.parent_hint[k >> 3] : kNoHint;
  const uint32_t* list = nullptr;
  uint32_t near = 0, info = kNoHint;
  int r = 0;
  if (k < lv.ncand) {
    int x, y, z;
    candidate_ijk(k, false, lv.res, lv.parents, x, y, z);
    float mn[3], mx[3];
    cube_box(x, y, z, lv.g, mn, mx);
    if (parent & kHintBit) {
      ShStack st{s_stack + threadIdx.x, 0};
      r = candidate_hit(nodes, tris, mn, mx, parent, st, info);
    } else {
      list = lv.parent_lists + parent;
      const uint32_t num = *list++;
      const GrownBox q = grown(mn, mx, lv.margin);
      for (uint32_t j = 0; j < num; ++j) {
        const float4* p = reinterpret_cast<const float4*>(tris + list[j]);
        if (meets(__ldg(p), __ldg(p + 1), __ldg(p + 2), q)) near |= 1u << j;
      }
      const float cx = box_centre(mn[0], mx[0]), cy = box_centre(mn[1], mx[1]), cz = box_centre(mn[2], mx[2]);
      const float hx = box_half(mn[0], mx[0]), hy = box_half(mn[1], mx[1]), hz = box_half(mn[2], mx[2]);
      for (uint32_t m = near; m; m &= m - 1u) {
        const uint32_t slot = list[__ffs((int)m) - 1];
        const float4* p = reinterpret_cast<const float4*>(tris + slot);
        if (sat_half(__ldg(p), __ldg(p + 1), __ldg(p + 2), cx, cy, cz, hx, hy, hz)) {
          info = slot | kHintBit;
          r = 1;
          break;
        }
      }
    }
  }
  if (kBuild) {
    const bool own = r == 1 && list != nullptr;
    const uint32_t num = (uint32_t)__popc(near);
    const uint32_t place = take_words(lv, own ? num + 1 : 0u);
    if (own && place != kNoHint) {
      uint32_t* o = lv.lists + place;
      *o++ = num;
      for (uint32_t m = near; m; m &= m - 1u) *o++ = list[__ffs((int)m) - 1];
      info = place;
    }
  }
  if (k < lv.ncand) put_decision(lv, k, r, info);
}

// the candidates whose walk outgrew its stack, one a thread
__global__ void octree_spill_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris, Level lv,
                                    int* __restrict__ overflow) {
  pdl_wait();
  const uint32_t m = *lv.nspill;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = lv.spill[t];
    int x, y, z;
    candidate_ijk(k, lv.first_level, lv.res, lv.parents, x, y, z);
    float mn[3], mx[3];
    cube_box(x, y, z, lv.g, mn, mx);
    LcStack st;
    st.sp = 0;
    uint32_t info = kNoHint;
    // a hint was tested in the level kernel; the walk decides
    const int r = candidate_hit(nodes, tris, mn, mx, kNoHint, st, info);
    if (r == 2) atomicExch(overflow, 1);
    lv.flags[k] = r == 1 ? 1u : 0u;
    lv.hit[k] = r == 1 ? 1 : 0;
    lv.ctri[k] = info;
  }
}

// stable compaction of the hit candidates (flags hold the exclusive scan
// after the scan pass; hit tested again from the candidate's own flag copy)
__global__ void octree_compact_kernel(int64_t ncand, bool first_level, int res, const int32_t* __restrict__ parents,
                                      const uint8_t* __restrict__ hit, const uint32_t* __restrict__ offs,
                                      const uint32_t* __restrict__ ctri, int32_t* __restrict__ out32,
                                      uint32_t* __restrict__ hint_out, int64_t* __restrict__ out64) {
  pdl_wait();
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ncand || !hit[k]) return;
  int x, y, z;
  candidate_ijk(k, first_level, res, parents, x, y, z);
  const int64_t o = offs[k];
  if (out64) {
    out64[3 * o] = x; out64[3 * o + 1] = y; out64[3 * o + 2] = z;
  } else {
    out32[3 * o] = x; out32[3 * o + 1] = y; out32[3 * o + 2] = z;
    hint_out[o] = ctri[k];
  }
}

// ---- Morton ------------------------------------------------------------------
__global__ void morton_encode_kernel(const int64_t* __restrict__ ijk, int64_t n, int64_t* __restrict__ out) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  // bits 0..20 of each coordinate (two's complement bits, like the
  // reference's shift-and-mask loop)
  const uint64_t x = (uint64_t)ijk[3 * i], y = (uint64_t)ijk[3 * i + 1], z = (uint64_t)ijk[3 * i + 2];
  out[i] = (int64_t)(spread3_21(x) | (spread3_21(y) << 1) | (spread3_21(z) << 2));
}

__global__ void morton_decode_kernel(const int64_t* __restrict__ m, int64_t n, int level, int64_t* __restrict__ ijk) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t v = (uint64_t)m[i];
  const int bits = level + 1 < 21 ? level + 1 : 21;
  const uint64_t mask = bits >= 64 ? ~0ull : ((1ull << bits) - 1);
  ijk[3 * i] = (int64_t)(compact3_21(v) & mask);
  ijk[3 * i + 1] = (int64_t)(compact3_21(v >> 1) & mask);
  ijk[3 * i + 2] = (int64_t)(compact3_21(v >> 2) & mask);
}

}  // namespace
}  // namespace a3d

using namespace a3d;

extern "C" int a3d_morton_encode(const int64_t* ijk, int64_t n, int64_t* morton, a3d_stream_t stream) {
  A3D_REQUIRE(n >= 0, A3D_ERR_ARGUMENT, "morton_encode: bad size");
  if (n == 0) return A3D_OK;
  A3D_PDL(morton_encode_kernel, dim3((unsigned)ceil_div(n, 256)), dim3(256), 0, (cudaStream_t)stream, ijk, n, morton);
  return A3D_OK;
}

extern "C" int a3d_morton_decode(const int64_t* morton, int64_t n, int level, int64_t* ijk, a3d_stream_t stream) {
  A3D_REQUIRE(n >= 0 && level >= 0, A3D_ERR_ARGUMENT, "morton_decode: bad argument");
  if (n == 0) return A3D_OK;
  A3D_PDL(morton_decode_kernel, dim3((unsigned)ceil_div(n, 256)), dim3(256), 0, (cudaStream_t)stream, morton, n, level,
          ijk);
  return A3D_OK;
}

extern "C" size_t a3d_aabb_hit_workspace_bytes(int64_t n) {
  Workspace ws(nullptr, 0);
  ws.take<uint32_t>(n);
  ws.take<uint32_t>(4);
  return ws.used + 256;
}

extern "C" int a3d_aabb_hit(const a3d_bvh_view* bvh, const float* box_min, const float* box_max, int64_t n,
                            uint8_t* hit, void* workspace, size_t workspace_bytes, a3d_stream_t stream) {
  cudaStream_t s = (cudaStream_t)stream;
  A3D_REQUIRE(bvh && bvh->nodes && bvh->tris, A3D_ERR_ARGUMENT, "aabb_hit: invalid bvh");
  A3D_REQUIRE(n >= 0 && n < (1ll << 32), A3D_ERR_ARGUMENT, "aabb_hit: bad size");
  if (n == 0) return A3D_OK;
  Workspace ws(workspace, workspace_bytes);
  uint32_t* spill = ws.take<uint32_t>(n);
  uint32_t* nspill = ws.take<uint32_t>(4);
  A3D_REQUIRE(workspace && ws.ok(), A3D_ERR_WORKSPACE, "aabb_hit: workspace too small");
  A3D_CUDA_TRY(cudaMemsetAsync(nspill, 0, 4 * sizeof(uint32_t), s));
  A3D_PDL(aabb_hit_kernel, dim3((unsigned)ceil_div(n, kSatThreads)), dim3(kSatThreads), 0, s,
          (const WideNode*)bvh->nodes, (const TriRec*)bvh->tris, box_min, box_max, n, hit, spill, nspill);
  A3D_PDL(aabb_hit_spill_kernel, dim3(num_sms() * 4), dim3(64), 0, s, (const WideNode*)bvh->nodes,
          (const TriRec*)bvh->tris, box_min, box_max, hit, spill, nspill, (int*)(nspill + 1));
  int ov = 0;
  A3D_CUDA_TRY(cudaMemcpyAsync(&ov, nspill + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
  A3D_CUDA_TRY(cudaStreamSynchronize(s));
  A3D_REQUIRE(ov == 0, A3D_ERR_OVERFLOW, "aabb_hit: traversal stack overflow");
  return A3D_OK;
}

namespace {
struct OctWs {
  int32_t* list_a;
  int32_t* list_b;
  uint32_t* hint_a;  // per entry of list_a: the triangle that hit it
  uint32_t* hint_b;
  uint32_t* ctri;    // per candidate: the triangle that hit it
  uint32_t* flags;
  uint8_t* hit;
  uint32_t* scan_tmp;
  uint32_t* spill;
  uint32_t* lists_a;  // triangle lists of one level and of the level before it
  uint32_t* lists_b;
  uint32_t* misc;  // [0] total, [1] spill count, [2] overflow, [3] words of lists
};
// words of a level's lists: two a voxel of capacity (a level that makes lists
// has about a quarter of the finest level's voxels, with 4 to 8 triangles each
// where triangles and voxels are of one size)
int64_t list_words(int64_t cap) { return 2 * cap < (1ll << 30) ? 2 * cap : (1ll << 30); }
size_t carve_oct(OctWs& w, Workspace& ws, int64_t cap) {
  const int64_t ncap = 8 * cap;
  w.list_a = ws.take<int32_t>(3 * cap);
  w.list_b = ws.take<int32_t>(3 * cap);
  w.hint_a = ws.take<uint32_t>(cap);
  w.hint_b = ws.take<uint32_t>(cap);
  w.ctri = ws.take<uint32_t>(ncap);
  w.flags = ws.take<uint32_t>(ncap);
  w.hit = ws.take<uint8_t>(ncap);
  w.scan_tmp = ws.take<uint32_t>((int64_t)scan_workspace_elems(ncap));
  w.spill = ws.take<uint32_t>(ncap);
  w.lists_a = ws.take<uint32_t>(list_words(cap));
  w.lists_b = ws.take<uint32_t>(list_words(cap));
  w.misc = ws.take<uint32_t>(8);
  return ws.used;
}
}  // namespace

namespace {
// The margin of the triangle lists' boxes, negative where no list is made.  A
// descendant's box reaches out of its ancestor's by the rounding of i * cell +
// lo and by unequal cells at both levels, and its SAT reaches sat_eps and the
// rounding of a centre, a half extent and a difference further: together below
// 1e-6 + 20 * 2^-24 M for coordinates up to M; 4e-6 (1 + M) is three times
// that.  Cells that are not
// halved from level to level (to 2^-22 of the grid), or are not finite, make no
// lists.
float list_margin(const float* lo, const float* cell, int min_level, int max_level) {
  double m = 0.0;
  for (int a = 0; a < 3; ++a) {
    const double extent = (double)cell[3 * min_level + a] * (double)(1 << min_level);
    if (!(extent > 0.0) || !(extent < 1e30) || !(fabs((double)lo[a]) < 1e30)) return -1.0f;
    for (int l = min_level; l <= max_level; ++l)
      if (!(fabs((double)cell[3 * l + a] * (double)(1 << l) - extent) <= extent * 0x1p-22)) return -1.0f;
    m = fmax(m, fabs((double)lo[a]) + extent);
  }
  return (float)(4e-6 * (1.0 + m));
}
}  // namespace

extern "C" size_t a3d_octree_workspace_bytes(int min_level, int max_level, int64_t cap) {
  (void)max_level;
  const int64_t first = 1ll << (3 * min_level);
  const int64_t c = cap > first ? cap : first;
  Workspace ws(nullptr, 0);
  OctWs w;
  return carve_oct(w, ws, c) + 256;
}

extern "C" int a3d_octree_traverse(const a3d_bvh_view* bvh, const float* grid_lo, const float* cell_sizes,
                                   int min_level, int max_level, int64_t* out_ijk, int64_t cap, int64_t* count_out,
                                   void* workspace, size_t workspace_bytes, a3d_stream_t stream) {
  cudaStream_t s = (cudaStream_t)stream;
  A3D_REQUIRE(bvh && bvh->nodes && bvh->tris, A3D_ERR_ARGUMENT, "octree: invalid bvh");
  A3D_REQUIRE(min_level >= 0 && max_level >= min_level && max_level <= 20, A3D_ERR_ARGUMENT,
              "octree: bad levels");
  A3D_REQUIRE(min_level <= 9, A3D_ERR_ARGUMENT, "octree: min_level above 9 (2^27 cubes) not supported");
  A3D_REQUIRE(count_out && grid_lo && cell_sizes, A3D_ERR_ARGUMENT, "octree: null argument");
  const int64_t first = 1ll << (3 * min_level);
  const int64_t c = cap > first ? cap : first;
  Workspace ws(workspace, workspace_bytes);
  OctWs w;
  carve_oct(w, ws, c);
  A3D_REQUIRE(workspace && ws.ok(), A3D_ERR_WORKSPACE, "octree: workspace too small");
  const WideNode* nodes = (const WideNode*)bvh->nodes;
  const TriRec* tris = (const TriRec*)bvh->tris;
  int64_t ncand = first;
  const int32_t* parents = nullptr;
  const uint32_t* parent_hint = nullptr;
  int32_t* next = w.list_a;
  uint32_t* next_hint = w.hint_a;
  uint32_t *lists = w.lists_a, *parent_lists = w.lists_b;
  bool have_lists = false;
  const float margin = list_margin(grid_lo, cell_sizes, min_level, max_level);
  *count_out = 0;
  for (int level = min_level; level <= max_level; ++level) {
    const bool first_level = level == min_level, last_level = level == max_level;
    const int res = 1 << level;
    LevelGeom g;
    for (int a = 0; a < 3; ++a) {
      g.lo[a] = grid_lo[a];
      g.cell[a] = cell_sizes[3 * level + a];
    }
    if (ncand > 8 * c) {
      *count_out = -1;
      A3D_REQUIRE(false, A3D_ERR_WORKSPACE, "octree: candidate capacity exceeded");
    }
    A3D_CUDA_TRY(cudaMemsetAsync(w.misc, 0, 8 * sizeof(uint32_t), s));
    const Level lv{ncand, first_level, res, parents, parent_hint, g, w.flags, w.hit, w.ctri, w.spill, w.misc + 1,
                   parent_lists, lists, (uint32_t)list_words(c), w.misc + 3, margin};
    const dim3 gk((unsigned)ceil_div(ncand, kSatThreads)), bk(kSatThreads);
    // Lists are collected at the first level that has, by the usual count of
    // four hit children a parent, at most eight triangles a hit voxel, where a
    // walk finds a whole list in few steps, or two on a level too small to fill
    // the chip, which waits for its longest walk.  (The voxel's box meets two or
    // three times that many triangles' boxes.)  The collecting walk costs more than
    // the one it replaces, so two levels must be left to gain by it.  (us, no lists
    // / eight triangles at every size and for one level / so: 128^3, 1,280 triangles
    // 260 / 240 / 249, 20,480 rough ones 513 / 555 / 520, 5,000 large ones 457 / 540
    // / 455; 512^3, 1,310,720 triangles 921 / 978 / 922.)  A tree of one node makes
    // none: its walk is as short as a list (1024^3, a cube's twelve triangles 752
    // us with lists, 684 without, 512^3 334 and 320; twenty of a sphere 440 and 432
    // at 1024^3).  Far from the origin and in tiny grids the margin is of a cell's
    // size and lists get longer: it counts with the cell, and takes half of one at
    // most (256^3, 81,920 triangles, a margin of one / two finest cells: 470 / 486 us
    // without lists, 514 / 618 when it did not count, 469 / 488 so; 512^3, 20,480
    // triangles: 742 / 749, 508 / 558, 508 / 559).
    const double near = margin / fmin(g.cell[0], fmin(g.cell[1], g.cell[2]));
    const bool collect = !have_lists && !first_level && level + 2 <= max_level && margin >= 0.0f &&
                         bvh->num_nodes > 1 && near <= 0.5 &&
                         (double)bvh->num_tris * (1.0 + near) * (1.0 + near) <=
                             (ncand >= kListFull ? 4.0 : 1.0) * (double)ncand;
    if (have_lists && last_level)
      A3D_PDL(octree_list_kernel<false>, gk, bk, 0, s, nodes, tris, lv);
    else if (have_lists)
      A3D_PDL(octree_list_kernel<true>, gk, bk, 0, s, nodes, tris, lv);
    else if (collect)
      A3D_PDL(octree_collect_kernel, gk, bk, 0, s, nodes, tris, lv);
    else
      A3D_PDL(octree_level_kernel, gk, bk, 0, s, nodes, tris, lv);
    have_lists = have_lists || collect;
    A3D_PDL(octree_spill_kernel, dim3(num_sms() * 4), dim3(64), 0, s, nodes, tris, lv, (int*)(w.misc + 2));
    A3D_TRY((device_exclusive_scan<uint32_t, uint32_t>(w.flags, w.flags, ncand, w.scan_tmp, w.misc, s)));
    uint32_t hm[3];
    A3D_CUDA_TRY(cudaMemcpyAsync(hm, w.misc, 3 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    A3D_CUDA_TRY(cudaStreamSynchronize(s));
    A3D_REQUIRE(hm[2] == 0, A3D_ERR_OVERFLOW, "octree: traversal stack overflow");
    const int64_t total = hm[0];
    const bool last = level == max_level;
    if (last) {
      *count_out = total;
      if (total > cap) {
        A3D_REQUIRE(false, A3D_ERR_WORKSPACE, "octree: output capacity exceeded");
      }
    } else if (total > c) {
      *count_out = -1;
      A3D_REQUIRE(false, A3D_ERR_WORKSPACE, "octree: level capacity exceeded");
    }
    A3D_PDL(octree_compact_kernel, dim3((unsigned)ceil_div(ncand, 256)), dim3(256), 0, s, ncand, first_level, res,
            parents, w.hit, w.flags, w.ctri, last ? nullptr : next, last ? nullptr : next_hint,
            last ? out_ijk : nullptr);
    if (last || total == 0) {
      if (!last) *count_out = 0;
      break;
    }
    parents = next;
    parent_hint = next_hint;
    next = (next == w.list_a) ? w.list_b : w.list_a;
    next_hint = (next_hint == w.hint_a) ? w.hint_b : w.hint_a;
    uint32_t* l = lists;
    lists = parent_lists;
    parent_lists = l;
    ncand = total * 8;
  }
  return A3D_OK;
}
