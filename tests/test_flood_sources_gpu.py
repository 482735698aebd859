"""Flood fills whose source lies on the faces, edges and corners of the bricks
that the relaxation works on (32 x 32 rows of 32 voxels): what only the seed
voxel touches, in its own brick or across a face, is filled like the rest.
Exact against the oracle's breadth-first fill, lists in their order."""

import numpy as np
import pytest
import torch

from atom3d_b200 import MeshBVH, OctreeIndexer, flood_fill_3d_sparse, sparse_flood_fill, synthetic

pytestmark = pytest.mark.gpu

NAMES = ["water", "dry", "tide", "dam", "dam_mask", "ext"]


def check(orc, dam, res, source, conn, padding=2):
    got = flood_fill_3d_sparse(torch.from_numpy(dam).cuda(), res, source=source, padding=padding, connectivity=conn)
    ref = orc.flood_fill_3d_sparse(dam, res, source=source, padding=padding, connectivity=conn)
    for a, b, name in zip(got, ref, NAMES):
        a = a.cpu().numpy()
        assert a.shape == b.shape and np.array_equal(a, b), (source, conn, name, a.shape, b.shape)


@pytest.mark.parametrize("conn", [6, 18, 26])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("at", [10, 31, 32, 50])
def test_source_in_a_one_voxel_tunnel(orc, conn, axis, at):
    dims = [12, 12, 12]
    dims[axis] = 61
    m = np.ones(dims, bool)
    tunnel = [5, 5, 5]
    tunnel[axis] = slice(10, 51)
    m[tuple(tunnel)] = False
    source = [5, 5, 5]
    source[axis] = at
    m[0, 0, 0] = m[tuple(d - 1 for d in dims)] = True
    check(orc, np.argwhere(m).astype(np.int64), 64, tuple(source), conn)


@pytest.mark.parametrize("conn", [6, 18, 26])
def test_source_whose_brick_has_no_other_free_voxel(orc, conn):
    """Every brick corner around (32, 32, 32), free voxels only across it."""
    for s in np.ndindex(2, 2, 2):
        m = np.ones((64, 64, 64), bool)
        source = tuple(31 + np.array(s))
        for axis in range(3):  # a run leaving the source's brick along each axis
            step = 1 if s[axis] else -1
            run = list(source)
            for _ in range(3):
                m[tuple(run)] = False
                run[axis] -= step
        check(orc, np.argwhere(m).astype(np.int64), 64, source, conn)


@pytest.mark.parametrize("conn", [6, 18, 26])
@pytest.mark.parametrize("density", [0.5, 0.7, 0.9])
def test_random_sources_in_random_dams(orc, conn, density):
    g = np.random.default_rng([conn, int(100 * density)])
    dims, res = np.array([66, 40, 70]), 96
    for k in range(24):
        m = g.random(dims) < density
        source = g.integers(0, dims)
        if k % 4:  # on a face, an edge or a corner of a brick
            edges = g.permutation(3)[:k % 4]
            source[edges] = g.integers(31, 33, len(edges))
        m[tuple(source)] = False
        m[0, 0, 0] = m[tuple(dims - 1)] = True
        check(orc, np.argwhere(m).astype(np.int64), res, tuple(int(c) for c in source), conn)


def test_default_source_in_the_last_corner_of_a_brick(orc):
    """k_ring 41 widens the volume by 31 beyond the crop on every side, so the
    crop's first voxel, the default source, is alone in its brick."""
    v, f = synthetic.displaced_sphere(3, 8, 0.05, 4)
    bounds = torch.tensor([[-3.6] * 3, [3.6] * 3], device="cuda")
    mesh = MeshBVH(v.cuda(), f.cuda())
    got = sparse_flood_fill(mesh, 128, connectivity=26, min_level=3, k_ring=41, bounds=bounds)
    dam = OctreeIndexer(max_level=7, bounds=bounds, device="cuda").octree_traverse(mesh, min_level=3).cpu().numpy()
    assert (dam.min(0) - 10 >= 31).all()
    ref = dict(zip(NAMES, orc.flood_fill_3d_sparse(dam, 128, padding=10, connectivity=26)))
    for name in ("water", "dry", "tide", "dam"):
        assert np.array_equal(got[name + "_ijk"].cpu().numpy(), ref[name]), name
    assert ref["water"].shape[0] > 10000
