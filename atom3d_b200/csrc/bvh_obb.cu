// Builds the oriented boxes of a finished wide BVH (bvh_obb.cuh) from its
// nodes and triangle records alone.
#include <math.h>

#include "bvh_obb.cuh"

namespace a3d {
namespace {

constexpr int kObbThreads = 256;
// subtrees above this have no oriented box: at that size a patch is curved
// and the axis-aligned box serves as well, and the pass over every level's
// triangles stays short
#ifndef A3D_OBB_MAX_TRIS
#define A3D_OBB_MAX_TRIS 4096
#endif
constexpr int64_t kObbMaxTris = A3D_OBB_MAX_TRIS;
constexpr int kMaxDescent = 64;  // wide levels of any tree the builder finishes

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) { return -warp_min(-v); }

// One warp per (node, child), bound by its L2 reads: every level of at most
// kObbMaxTris triangles reads all records twice (223 us for 1,310,720
// triangles, 3% of the build it follows).  A subtree's triangles are one range of the
// records: the range runs from the first triangle of its leftmost leaf to
// the last of its rightmost one.
__global__ void __launch_bounds__(kObbThreads)
    obb_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris, int64_t num_nodes,
               const int64_t* __restrict__ num_nodes_dev, int64_t num_tris, ObbNode* __restrict__ out) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  int64_t count = num_nodes;
  if (num_nodes_dev != nullptr && *num_nodes_dev < count) count = *num_nodes_dev;
  const int64_t warps = (int64_t)gridDim.x * (kObbThreads / 32);
  for (int64_t w = ((int64_t)blockIdx.x * kObbThreads + threadIdx.x) >> 5; w < 4 * count; w += warps) {
    const WideNode* nd = nodes + (w >> 2);
    const int c = (int)(w & 3);
    ObbChild res{512u | (512u << 10) | (513u << 20), -INFINITY, INFINITY, -INFINITY, INFINITY, -INFINITY, INFINITY,
                 0.f};
    if (c < (int)(nd->meta >> 24)) {
      const uint32_t r = nd->ref[c];
      uint32_t a = r, b = r;
      for (int k = 0; k < kMaxDescent && !ref_is_leaf(a) && a < (uint64_t)count; ++k) a = nodes[a].ref[0];
      for (int k = 0; k < kMaxDescent && !ref_is_leaf(b) && b < (uint64_t)count; ++k) {
        const int nch = (int)(nodes[b].meta >> 24);
        b = nodes[b].ref[nch > 0 ? nch - 1 : 0];
      }
      const int64_t first = leaf_first(a), last = (int64_t)leaf_first(b) + leaf_count(b);
      if (ref_is_leaf(a) && ref_is_leaf(b) && first < last && last <= num_tris && last - first <= kObbMaxTris) {
        // direction: the sum of the triangles' area vectors
        float nx = 0.f, ny = 0.f, nz = 0.f;
        for (int64_t i = first + lane; i < last; i += 32) {
          const float4 A = tris[i].a, B = tris[i].b, C = tris[i].c;
          const float ux = B.x - A.x, uy = B.y - A.y, uz = B.z - A.z;
          const float vx = C.x - A.x, vy = C.y - A.y, vz = C.z - A.z;
          nx += uy * vz - uz * vy;
          ny += uz * vx - ux * vz;
          nz += ux * vy - uy * vx;
        }
        nx = warp_sum(nx);
        ny = warp_sum(ny);
        nz = warp_sum(nz);
        const float m = fmaxf(fabsf(nx), fmaxf(fabsf(ny), fabsf(nz)));
        if (m > 0.f && m < INFINITY) {
          const uint32_t ix = (uint32_t)(__float2int_rn(nx / m * 511.f) + 512),
                         iy = (uint32_t)(__float2int_rn(ny / m * 511.f) + 512),
                         iz = (uint32_t)(__float2int_rn(nz / m * 511.f) + 512);
          const uint32_t dir = ix | (iy << 10) | (iz << 20);
          float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY}, big = 0.f;
          for (int64_t i = first + lane; i < last; i += 32) {
            const float4 P[3] = {tris[i].a, tris[i].b, tris[i].c};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const float qx = P[k].x - nd->ox, qy = P[k].y - nd->oy, qz = P[k].z - nd->oz;
              float q[3];
              obb_frame(dir, qx, qy, qz, q[0], q[1], q[2]);
#pragma unroll
              for (int x = 0; x < 3; ++x) {
                lo[x] = fminf(lo[x], q[x]);
                hi[x] = fmaxf(hi[x], q[x]);
              }
              const float g = fabsf(qx) + fabsf(qy) + fabsf(qz);
              big = g <= big ? big : g;  // keeps a NaN
            }
          }
          // an infinite or NaN vertex: no box
          const bool finite = __all_sync(0xffffffffu, big < INFINITY);
          big = kObbSlack * warp_max(big);  // the projections' rounding
#pragma unroll
          for (int x = 0; x < 3; ++x) {
            lo[x] = warp_min(lo[x]) - big;
            hi[x] = warp_max(hi[x]) + big;
          }
          if (finite) res = ObbChild{dir, lo[0], hi[0], lo[1], hi[1], lo[2], hi[2], 0.f};
        }
      }
    }
    if (lane == 0) out[w >> 2].child[c] = res;
  }
}

}  // namespace
}  // namespace a3d

using namespace a3d;

extern "C" int a3d_bvh_obbs(const void* nodes, const void* tris, int64_t num_nodes, const int64_t* num_nodes_device,
                            int64_t num_tris, void* obbs_out, a3d_stream_t stream) {
  A3D_REQUIRE(nodes && tris && obbs_out && num_nodes > 0 && num_tris > 0, A3D_ERR_ARGUMENT, "bvh_obbs: invalid bvh");
  A3D_REQUIRE(((uintptr_t)obbs_out & 15) == 0, A3D_ERR_ARGUMENT, "bvh_obbs: boxes must be 16-B aligned");
  const int64_t want = ceil_div(4 * num_nodes, kObbThreads / 32);
  const int64_t cap = (int64_t)num_sms() * 32;
  A3D_PDL(obb_kernel, dim3((unsigned)(want < cap ? want : cap)), dim3(kObbThreads), 0, (cudaStream_t)stream,
          (const WideNode*)nodes, (const TriRec*)tris, num_nodes, num_nodes_device, num_tris, (ObbNode*)obbs_out);
  return A3D_OK;
}
