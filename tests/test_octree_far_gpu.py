"""Octree descents of grids far from the origin and of tiny ones, on both sides
of the line where the margin of the triangle lists is half a cell, against a
descent that asks one any-hit query per candidate."""

import pytest
import torch

from atom3d_b200 import MeshBVH, OctreeIndexer, synthetic

pytestmark = pytest.mark.gpu

CORNERS = torch.tensor([[c & 1, (c >> 1) & 1, (c >> 2) & 1] for c in range(8)], dtype=torch.int64)


@pytest.mark.parametrize("scale, offset", [(1.0, 500.0), (1.0, 4500.0), (1.0, 4900.0), (1.0, 9000.0), (1e-2, 0.0),
                                           (2.5e-4, 0.0), (2e-4, 0.0), (1e-5, 0.0)])
def test_far_and_tiny_grids(scale, offset):
    # the last level that may collect has 2^6 cells of 2.4 / 64; the margin,
    # 4e-6 (1 + offset + 1.2), is half of one at an offset of 4,685, or 4e-6 at a
    # scale of 2.13e-4
    v, f = synthetic.displaced_sphere(4, 8, 0.05, 7)
    mesh = MeshBVH((v * scale + offset).cuda(), f.cuda())
    bounds = torch.tensor([[-1.2] * 3, [1.2] * 3]) * scale + offset
    octree = OctreeIndexer(max_level=8, bounds=bounds.cuda(), device="cuda")
    got = octree.octree_traverse(mesh, min_level=3)
    ax = torch.arange(8, device="cuda")
    cand = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    for level in range(3, 9):
        if level > 3:
            cand = (2 * cand[:, None, :] + CORNERS.cuda()[None]).reshape(-1, 3)
        lo, hi = octree.cube_aabb_level(cand, level)
        cand = cand[mesh.intersect_aabb(lo, hi, mode=0).hit]
    assert cand.shape[0] > 0 and torch.equal(got, cand)
