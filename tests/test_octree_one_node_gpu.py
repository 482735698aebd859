"""Octree descents of trees of one node, which make no triangle lists, against
the same tree with a node count in its view for which lists are made."""

import pytest
import torch

from atom3d_b200 import MeshBVH, OctreeIndexer, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tris", [1, 2, 8, 12])
@pytest.mark.parametrize("levels", [(0, 3), (2, 6), (4, 8)])
def test_walks_against_lists(tris, levels):
    g = torch.Generator().manual_seed(tris)
    v = (1.6 * torch.rand(tris, 3, 3, generator=g) - 0.8).reshape(-1, 3)
    mesh = MeshBVH(v.cuda(), torch.arange(3 * tris, dtype=torch.int32).reshape(-1, 3).cuda())
    view = mesh._bvh.view
    if view.num_nodes != 1:
        assert tris > 8
        pytest.skip("the builder made more than one node of these triangles")
    bounds = torch.tensor([[-1.0, -1.1, -1.3], [1.2, 1.0, 1.0]], device="cuda")
    octree = OctreeIndexer(max_level=levels[1], bounds=bounds, device="cuda")
    got = octree.octree_traverse(mesh, min_level=levels[0])
    general = _lib.BvhView.from_buffer_copy(view)
    general.num_nodes = 2
    mesh._bvh._view = general
    ref = octree.octree_traverse(mesh, min_level=levels[0])
    assert got.shape[0] > 0 and torch.equal(got, ref)
