"""The pair walk of MeshBVH.intersect_aabb where warps go back and forth between
steps that compare the triangles' own boxes first and dense ones that do not.
Against the oracle's brute force; within a box the faces come in tree order."""

import numpy as np
import pytest
import torch

from atom3d_b200 import MeshBVH

pytestmark = pytest.mark.gpu


def _check(orc, mesh, v, f, mn, mx):
    r = mesh.intersect_aabb(torch.from_numpy(mn).cuda(), torch.from_numpy(mx).cuda(), mode=1)
    ref = orc.aabb_pairs(v, f, mn, mx, mode=1)
    a, fc = r.aabb_ids.cpu().numpy(), r.face_ids.cpu().numpy()
    assert np.all(np.diff(a) >= 0)
    o = np.lexsort((fc, a))
    assert np.array_equal(a[o], ref["aabb_ids"]) and np.array_equal(fc[o], ref["face_ids"])
    place = np.empty(len(f), dtype=np.int64)
    place[mesh._bvh.tris.view(torch.int32).view(len(f), 16)[:, 3].cpu().numpy()] = np.arange(len(f))
    same = a[1:] == a[:-1]
    assert np.all(place[fc[1:]][same] > place[fc[:-1]][same])
    return np.bincount(a, minlength=len(mn))


@pytest.mark.parametrize("n", [1, 33, 5000])
def test_dense_and_sparse_leaves(orc, n):
    # a cluster far smaller than the boxes, in which every leaf's triangles
    # pass, among scattered triangles, of which few do
    g = np.random.default_rng(n)
    t = 3000
    knot = 0.3 + 1e-3 * g.uniform(-1, 1, (t // 2, 1, 3)) + 2e-5 * g.normal(size=(t // 2, 3, 3))
    wide = g.uniform(-1, 1, (t - t // 2, 1, 3)) + 0.05 * g.normal(size=(t - t // 2, 3, 3))
    v = np.concatenate([knot, wide]).astype(np.float32).reshape(-1, 3)
    f = np.arange(3 * t, dtype=np.int32).reshape(-1, 3)
    mesh = MeshBVH(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda())
    c = np.where(g.random((n, 1)) < 0.1, 0.3 + 2e-3 * g.normal(size=(n, 3)), g.uniform(-1, 1, (n, 3)))
    c[0] = 0.3
    h = np.exp(g.uniform(np.log(5e-4), np.log(0.05), (n, 1)))
    h[0] = 0.01
    mn, mx = (c - h).astype(np.float32), (c + h).astype(np.float32)
    counts = _check(orc, mesh, v, f, mn, mx)
    assert counts[0] >= t // 2
    assert n < 100 or (np.median(counts) < 20 and (counts > t // 4).any())
