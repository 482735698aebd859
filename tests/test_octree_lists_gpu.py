"""The octree descent's triangle lists against a descent that asks one any-hit
query per candidate (MeshBVH.intersect_aabb mode 0, which walks the tree):
meshes whose voxels meet few triangles, more than a list holds, and both side
by side, on grids at and far from the origin; voxels and order equal."""

import numpy as np
import pytest
import torch

from atom3d_b200 import MeshBVH, OctreeIndexer, synthetic

pytestmark = pytest.mark.gpu

CORNERS = torch.tensor([[c & 1, (c >> 1) & 1, (c >> 2) & 1] for c in range(8)], dtype=torch.int64)


def _mesh(kind):
    v, f = synthetic.displaced_sphere(3, 8, 0.05, 7)
    v, f = v.numpy() * 0.8, f.numpy()
    if kind == "even":
        return v, f
    g = np.random.default_rng(3)
    # a knot of small triangles, far more than a list holds in its voxels, and
    # a few triangles across the grid
    n = 6000
    c = g.normal(0, 0.02, (n, 1, 3)) + np.array([0.3, 0.2, -0.1])
    knot = (c + g.normal(0, 0.004, (n, 3, 3))).reshape(-1, 3)
    wide = g.uniform(-0.9, 0.9, (24, 3)).repeat(1, axis=0)
    parts = [knot, wide] if kind == "knot" else [v, knot, wide]
    faces, base = [], 0
    for p in parts:
        faces.append((f if p is v else np.arange(len(p)).reshape(-1, 3)) + base)
        base += len(p)
    return np.concatenate(parts), np.concatenate(faces)


def _descent(octree, mesh, min_level, max_level):
    n = 1 << min_level
    ax = torch.arange(n, device="cuda")
    cand = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    for level in range(min_level, max_level + 1):
        if level > min_level:
            cand = (2 * cand[:, None, :] + CORNERS.cuda()[None]).reshape(-1, 3)
        lo, hi = octree.cube_aabb_level(cand, level)
        cand = cand[mesh.intersect_aabb(lo, hi, mode=0).hit]
    return cand


@pytest.mark.parametrize("kind", ["even", "knot", "both"])
@pytest.mark.parametrize("offset", [0.0, 37.0])
@pytest.mark.parametrize("levels", [(2, 3), (3, 6), (2, 8)])
def test_lists_against_walks(kind, offset, levels):
    v, f = _mesh(kind)
    v = torch.from_numpy((v + offset).astype(np.float32)).cuda()
    mesh = MeshBVH(v, torch.from_numpy(f.astype(np.int32)).cuda())
    bounds = torch.tensor([[-1.0, -1.1, -1.3], [1.2, 1.0, 1.0]]) + offset
    octree = OctreeIndexer(max_level=levels[1], bounds=bounds.cuda(), device="cuda")
    got = octree.octree_traverse(mesh, min_level=levels[0])
    ref = _descent(octree, mesh, *levels)
    assert ref.shape[0] > 0 and torch.equal(got, ref)
