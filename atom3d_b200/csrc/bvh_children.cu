// Builds the child records of a finished wide BVH (bvh_children.cuh) from its
// nodes and triangle records alone.
#include <math.h>

#include "bvh_children.cuh"

namespace a3d {
namespace {

constexpr int kChildThreads = 256;
// subtrees above this have no disc: at that size a patch is curved and the
// axis-aligned box serves as well, and the pass over every level's triangles
// stays short
constexpr int64_t kDiscMaxTris = 4096;
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
// kDiscMaxTris triangles reads all records three times.  A subtree's triangles
// are one range of the records: from the first triangle of its leftmost leaf
// to the last of its rightmost one.
__global__ void __launch_bounds__(kChildThreads)
    child_kernel(const WideNode* __restrict__ nodes, const TriRec* __restrict__ tris, int64_t num_nodes,
                 const int64_t* __restrict__ num_nodes_dev, bool by_count, int64_t num_tris, void* children) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  // num_nodes is a capacity when the count is on the device.  The records are
  // laid out for it (nodes past it have no boxes and no disc, the leaves under
  // them still do), or, by_count, for the count, and left out if they do not fit
  const int64_t count = num_nodes_dev != nullptr ? *num_nodes_dev : num_nodes;
  if (by_count) {
    if (count > num_nodes) return;
    num_nodes = count;
  }
  const ChildRecs cr(children, num_nodes);
  BoxRec* __restrict__ boxes = const_cast<BoxRec*>(cr.boxes);
  DiscRec* __restrict__ node_discs = const_cast<DiscRec*>(cr.node_discs);
  DiscRec* __restrict__ leaf_discs = const_cast<DiscRec*>(cr.leaf_discs);
  const DiscRec no_disc{0.f, 0.f, 0.f, INFINITY, 0.f, 0.f, 1.f, INFINITY};
  if (blockIdx.x == 0 && threadIdx.x == 0) leaf_discs[num_tris] = no_disc;
  const int64_t warps = (int64_t)gridDim.x * (kChildThreads / 32);
  for (int64_t w = ((int64_t)blockIdx.x * kChildThreads + threadIdx.x) >> 5; w < 4 * count; w += warps) {
    const WideNode* nd = nodes + (w >> 2);
    const int c = (int)(w & 3);
    BoxRec box{INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY, 0xffffffffu, 0u};
    DiscRec disc = no_disc;
    int64_t leaf_at = -1, node_at = -1;
    if (c < (int)(nd->meta >> 24)) {
      const uint32_t r = nd->ref[c];
      const float sx = __uint_as_float((nd->meta & 0xffu) << 23);
      const float sy = __uint_as_float(((nd->meta >> 8) & 0xffu) << 23);
      const float sz = __uint_as_float(((nd->meta >> 16) & 0xffu) << 23);
      box.lx = dequant(nd->q[0], c, sx, nd->ox);
      box.ly = dequant(nd->q[1], c, sy, nd->oy);
      box.lz = dequant(nd->q[2], c, sz, nd->oz);
      box.hx = dequant(nd->q[3], c, sx, nd->ox);
      box.hy = dequant(nd->q[4], c, sy, nd->oy);
      box.hz = dequant(nd->q[5], c, sz, nd->oz);
      box.ref = (ref_is_leaf(r) ? leaf_first(r) + leaf_count(r) <= (uint64_t)num_tris : r < (uint64_t)count)
                    ? r
                    : make_leaf_ref((uint32_t)num_tris, 1u);
      for (int x = 1; x < 4; ++x) box.ties |= nd->ref[c ^ x] < r ? 1u << (x - 1) : 0u;
      if (ref_is_leaf(r)) {
        if (leaf_first(r) < (uint64_t)num_tris) leaf_at = leaf_first(r);
      } else if (r < (uint64_t)num_nodes) {
        node_at = r;
      }
      uint32_t a = r, b = r;
      for (int k = 0; k < kMaxDescent && !ref_is_leaf(a) && a < (uint64_t)count; ++k) a = nodes[a].ref[0];
      for (int k = 0; k < kMaxDescent && !ref_is_leaf(b) && b < (uint64_t)count; ++k) {
        const int nch = (int)(nodes[b].meta >> 24);
        b = nodes[b].ref[nch > 0 ? nch - 1 : 0];
      }
      const int64_t first = leaf_first(a), last = (int64_t)leaf_first(b) + leaf_count(b);
      if (ref_is_leaf(a) && ref_is_leaf(b) && first < last && last <= num_tris && last - first <= kDiscMaxTris) {
        // normal: the sum of the triangles' area vectors
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
          nx /= m; ny /= m; nz /= m;
          const float len = sqrtf(nx * nx + ny * ny + nz * nz);
          nx /= len; ny /= len; nz /= len;
          // two tangents (Duff et al. 2017, "Building an Orthonormal Basis, Revisited")
          const float sg = copysignf(1.f, nz);
          const float ta = -1.f / (sg + nz), tb = nx * ny * ta;
          const float ux = 1.f + sg * nx * nx * ta, uy = sg * tb, uz = -sg * nx;
          const float vx = tb, vy = sg + ny * ny * ta, vz = -ny;
          // centre: the middle of the extents along the normal and the tangents
          const float ox = nd->ox, oy = nd->oy, oz = nd->oz;
          float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
          for (int64_t i = first + lane; i < last; i += 32) {
            const float4 P[3] = {tris[i].a, tris[i].b, tris[i].c};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const float qx = P[k].x - ox, qy = P[k].y - oy, qz = P[k].z - oz;
              const float q[3] = {nx * qx + ny * qy + nz * qz, ux * qx + uy * qy + uz * qz,
                                  vx * qx + vy * qy + vz * qz};
#pragma unroll
              for (int x = 0; x < 3; ++x) {
                lo[x] = fminf(lo[x], q[x]);
                hi[x] = fmaxf(hi[x], q[x]);
              }
            }
          }
          float mid[3];
#pragma unroll
          for (int x = 0; x < 3; ++x) mid[x] = 0.5f * (warp_min(lo[x]) + warp_max(hi[x]));
          const float cx = ox + (mid[0] * nx + mid[1] * ux + mid[2] * vx);
          const float cy = oy + (mid[0] * ny + mid[1] * uy + mid[2] * vy);
          const float cz = oz + (mid[0] * nz + mid[1] * uz + mid[2] * vz);
          // radius and half thickness about that centre
          float rho2 = 0.f, h = 0.f, big = 0.f;
          for (int64_t i = first + lane; i < last; i += 32) {
            const float4 P[3] = {tris[i].a, tris[i].b, tris[i].c};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const float qx = P[k].x - cx, qy = P[k].y - cy, qz = P[k].z - cz;
              const float s = nx * qx + ny * qy + nz * qz;
              const float lx = qx - s * nx, ly = qy - s * ny, lz = qz - s * nz;
              rho2 = fmaxf(rho2, lx * lx + ly * ly + lz * lz);
              h = fmaxf(h, fabsf(s));
              const float g = fabsf(qx) + fabsf(qy) + fabsf(qz);
              big = g <= big ? big : g;  // keeps a NaN
            }
          }
          // an infinite or NaN vertex (or a centre that is one): no disc
          const bool finite = __all_sync(0xffffffffu, big < INFINITY);
          big = 2.f * kDiscSlack * warp_max(big);  // the projections' rounding
          rho2 = warp_max(rho2);
          h = warp_max(h);
          if (finite) {
            disc = DiscRec{cx, cy, cz, sqrtf(rho2) + big, nx, ny, nz, h + big};
          }
        }
      }
    }
    if (lane == 0) {
      if (w < 4 * num_nodes) boxes[w] = box;
      if (leaf_at >= 0) leaf_discs[leaf_at] = disc;
      if (node_at >= 0) node_discs[node_at] = disc;
    }
  }
}

}  // namespace

int launch_children(const void* nodes, const void* tris, int64_t num_nodes, const int64_t* num_nodes_device,
                    bool by_count, int64_t num_tris, void* children_out, cudaStream_t s) {
  A3D_REQUIRE(((uintptr_t)children_out & 31) == 0, A3D_ERR_ARGUMENT, "bvh_children: records must be 32-B aligned");
  const int64_t want = ceil_div(4 * num_nodes, kChildThreads / 32);
  const int64_t cap = (int64_t)num_sms() * 32;
  A3D_PDL(child_kernel, dim3((unsigned)(want < cap ? want : cap)), dim3(kChildThreads), 0, s, (const WideNode*)nodes,
          (const TriRec*)tris, num_nodes, num_nodes_device, by_count, num_tris, children_out);
  return A3D_OK;
}

}  // namespace a3d

using namespace a3d;

extern "C" size_t a3d_bvh_children_bytes(int64_t num_nodes, int64_t num_tris) {
  return (size_t)(num_nodes > 0 ? num_nodes : 0) * (4 * sizeof(BoxRec) + sizeof(DiscRec)) +
         (size_t)(num_tris > 0 ? num_tris + 1 : 1) * sizeof(DiscRec);
}

extern "C" int a3d_bvh_children(const void* nodes, const void* tris, int64_t num_nodes, const int64_t* num_nodes_device,
                             int64_t num_tris, void* children_out, a3d_stream_t stream) {
  A3D_REQUIRE(nodes && tris && children_out && num_nodes > 0 && num_tris > 0, A3D_ERR_ARGUMENT,
              "bvh_children: invalid bvh");
  return launch_children(nodes, tris, num_nodes, num_nodes_device, false, num_tris, children_out, (cudaStream_t)stream);
}
