// Oriented boxes of the wide BVH's children: a second, much tighter lower
// bound on the distance to a subtree of a smooth surface.
//
// A child's axis-aligned box around a patch of h x h surface is as thick as
// the patch is wide wherever the surface is not axis-aligned, so a query at
// distance D meets every leaf within about sqrt(2 D h) of its closest point.
// A box along the patch's mean normal is only h^2 / (8 R) thick (R the radius
// of curvature), and the query meets little more than the leaves around the
// closest point.  16.8M mixed queries against 1.31M triangles: triangle tests
// 383 -> 38 and node visits 85 -> 31 a query, the traversal 144 -> 45 ms; on a
// surface with vertex noise of a quarter edge (20,480 triangles, 100,000
// queries) 54 -> 29 tests and 1.09 -> 0.63 ms.  (Two planes across the mean
// normal alone leave 313 tests: a neighbouring patch's planes slope towards a
// query outside, so the bound needs the sides of the box too.)
//
// ObbNode (128 B), one per wide node; child c is two 16-B words:
//   uint32 dir   direction d of the mean normal, 10 bits per axis biased by
//                512 (x | y << 10 | z << 20), components -511..511
//   float n0, n1, u0, u1, v0, v1   extent of the child's vertices, relative
//                to the node's origin, along the frame (n, u, v) that
//                obb_frame makes of d, widened by their rounding error;
//                -inf / +inf when the child has no oriented box
// The frame is built from the decoded integer vector on both sides, so
// rounding the direction costs thickness, never validity.
#pragma once

#include "a3d_common.cuh"
#include "bvh_layout.cuh"

namespace a3d {

struct __align__(16) ObbChild {
  uint32_t dir;
  float n0, n1, u0;
  float u1, v0, v1, pad;
};
struct __align__(16) ObbNode {
  ObbChild child[4];
};
static_assert(sizeof(ObbNode) == A3D_BVH_OBB_BYTES, "oriented-box records are 128 bytes");

// 10-bit field `shift` of a direction word as a float (-512..511), without
// the conversion unit: the field in the mantissa of 2^23, less 2^23 + 512
__device__ __forceinline__ float obb_axis(uint32_t w, int shift) {
  return __uint_as_float(((w >> shift) & 0x3ffu) | 0x4B000000u) - 8389120.0f;
}

// (n, u, v) coordinates of q in the frame of direction word `dir`: n = d/|d|,
// u and v the branchless orthonormal basis of Duff et al. 2017 ("Building an
// Orthonormal Basis, Revisited")
__device__ __forceinline__ void obb_frame(uint32_t dir, float qx, float qy, float qz, float& qn, float& qu,
                                          float& qv) {
  const float dx = obb_axis(dir, 0), dy = obb_axis(dir, 10), dz = obb_axis(dir, 20);
  const float il = rsqrtf(dx * dx + dy * dy + dz * dz);
  const float nx = dx * il, ny = dy * il, nz = dz * il;
  const float sg = copysignf(1.f, nz);
  const float a = -__fdividef(1.f, sg + nz);
  const float b = nx * ny * a;
  qn = nx * qx + ny * qy + nz * qz;
  qu = (1.f + sg * nx * nx * a) * qx + sg * b * qy - sg * nx * qz;
  qv = b * qx + (sg + ny * ny * a) * qy - ny * qz;
}

// Rounding allowance of an oriented distance, per axis and relative to |q|_1
// (q the query relative to the node's origin): the frame's and the products'
// own error (about 10 ulp) and that of the triangle tests the bound stands in
// for (the point they evaluate lies in the triangle to a few ulp of the
// distance plus the triangle's size)
constexpr float kObbSlack = 3e-6f;

// lower bound on the squared distance from the query (q relative to the
// node's origin) to any triangle of the child, as its triangle test would
// evaluate it; 0 when the box says nothing (NaN queries included)
__device__ __forceinline__ float obb_dist_sq(const ObbChild* oc, float qx, float qy, float qz) {
  const float4 w0 = __ldg(reinterpret_cast<const float4*>(oc));
  const float4 w1 = __ldg(reinterpret_cast<const float4*>(oc) + 1);
  float n, u, v;
  obb_frame(__float_as_uint(w0.x), qx, qy, qz, n, u, v);
  const float s = kObbSlack * (fabsf(qx) + fabsf(qy) + fabsf(qz));
  const float dn = fmaxf(fmaxf(w0.y - n, n - w0.z) - s, 0.f);
  const float du = fmaxf(fmaxf(w0.w - u, u - w1.x) - s, 0.f);
  const float dv = fmaxf(fmaxf(w1.y - v, v - w1.z) - s, 0.f);
  return (dn * dn + du * du + dv * dv) * (1.f - kObbSlack);
}

}  // namespace a3d
