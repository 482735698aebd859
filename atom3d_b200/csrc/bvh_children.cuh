// Child records of the wide BVH for the closest-point traversal: each child's
// box decoded, its reference, and a disc about its triangles, a second and
// much tighter lower bound on the distance to a subtree of a smooth surface.
//
// A child's axis-aligned box around a patch of h x h surface is as thick as
// the patch is wide wherever the surface is not axis-aligned, so a query at
// distance D meets every leaf within about sqrt(2 D h) of its closest point.
// A flat disc (a cylinder) along the patch's mean normal is only h^2 / (8 R)
// thick (R the radius of curvature), and the query meets little more than the
// leaves around the closest point.  16.8M mixed queries against 1.31M
// triangles: triangle tests 383 -> 38 and node visits 85 -> 26 a query.  (An
// oriented box in a frame made of the normal alone bounds no tighter on
// average, 1 + 2/pi of a square patch's area against pi/2, and costs 58
// instead of 25 instructions; two planes across the normal alone leave 313
// tests, because a neighbouring patch's planes slope towards a query outside.)
//
// BoxRec (32 B, one load), four per wide node in child order, so that the four
// lanes of a query read 128 contiguous bytes:
//   float lo[3], hi[3]      the quantised box's decoded corners (the values
//                           dequant() gives, so box distances are the same)
//   uint32 ref, ties        the node's reference, 0xffffffff for no child;
//                           bit x - 1 set when sibling c ^ x's is smaller
//                           (a reference to no node or triangle of the tree
//                           is stored as the leaf of one triangle at num_tris)
// DiscRec (32 B, one load), one per wide node and one per leaf, the latter at
// the place of the leaf's first triangle, and one more at num_tris:
//   float cx, cy, cz, rho   centre and radius of the disc
//   float nx, ny, nz, h     unit normal and half thickness
// rho and h are widened by their rounding error; rho = +inf for no disc.
// The buffer holds the boxes, the nodes' discs and the leaves' discs in turn.
#pragma once

#include "a3d_common.cuh"
#include "bvh_layout.cuh"

namespace a3d {

struct __align__(32) BoxRec {
  float lx, ly, lz, hx;
  float hy, hz;
  uint32_t ref, ties;
};
struct __align__(32) DiscRec {
  float cx, cy, cz, rho;
  float nx, ny, nz, h;
};
static_assert(sizeof(BoxRec) == 32 && sizeof(DiscRec) == 32, "child records are 32 bytes");

struct ChildRecs {
  const BoxRec* boxes;         // 4 per node
  const DiscRec* node_discs;   // by node
  const DiscRec* leaf_discs;   // by the leaf's first triangle
  __host__ __device__ ChildRecs(const void* p, int64_t num_nodes)
      : boxes(static_cast<const BoxRec*>(p)),
        node_discs(reinterpret_cast<const DiscRec*>(boxes + 4 * num_nodes)),
        leaf_discs(node_discs + num_nodes) {}
};

// Launches the pass that writes the records of a finished tree.  num_nodes: the
// tree's nodes, or a capacity with the count in *num_nodes_device; laid out for
// num_nodes or, by_count, for the count (nothing is written past the capacity).
int launch_children(const void* nodes, const void* tris, int64_t num_nodes, const int64_t* num_nodes_device,
                    bool by_count, int64_t num_tris, void* children_out, cudaStream_t s);

// Rounding allowance of a disc distance, relative to |q| (q the query
// relative to the disc's centre): the bound's own error (about 10 ulp) and
// that of the triangle tests it stands in for (the point they evaluate lies
// in the triangle to a few ulp of the distance plus the triangle's size).
constexpr float kDiscSlack = 3e-6f;

// lower bound on the squared distance from p to any triangle of the child, as
// its triangle test would evaluate it; 0 when the disc says nothing (NaN and
// infinite queries included)
__device__ __forceinline__ float disc_dist_sq(const DiscRec* rec, float px, float py, float pz) {
  float4 c, n;
  ldg256(rec, c, n);
  const float qx = px - c.x, qy = py - c.y, qz = pz - c.z;
  const float s = n.x * qx + n.y * qy + n.z * qz;
  const float m = qx * qx + qy * qy + qz * qz;
  const float slack = kDiscSlack * (fabsf(qx) + fabsf(qy) + fabsf(qz));
  // squared distance from the axis, less the error of the subtraction
  const float l2 = fmaxf((1.f - kDiscSlack) * m - s * s, 1e-36f);
  const float lat = fmaxf(l2 * rsqrtf(l2) - c.w - slack, 0.f);
  const float dn = fmaxf(fabsf(s) - n.w - slack, 0.f);
  return (dn * dn + lat * lat) * (1.f - kDiscSlack);
}

}  // namespace a3d
