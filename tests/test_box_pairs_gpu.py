"""The pair walk of MeshBVH.intersect_aabb at its edges: box counts around a
warp and its refills, boxes with as many pairs as are kept and one more, boxes
that meet the whole mesh, and a deep tree; against the oracle's brute force
(pairs as sets per box, clip outputs bit for bit) and against themselves in
other batches (the order within a box is the tree's)."""

import numpy as np
import pytest
import torch

from atom3d_b200 import MeshBVH, synthetic

pytestmark = pytest.mark.gpu

KEPT = 8  # pairs a box keeps from the count pass


def _boxes(n, seed):
    g = np.random.default_rng(seed)
    c = g.normal(size=(n, 3))
    c = c / np.linalg.norm(c, axis=1, keepdims=True) * g.uniform(0.9, 1.1, (n, 1))
    h = np.exp(g.uniform(np.log(0.01), np.log(0.3), (n, 1))) * g.uniform(0.5, 1.5, (n, 3))
    mn, mx = (c - h).astype(np.float32), (c + h).astype(np.float32)
    mn[n // 2], mx[n // 2] = -2.0, 2.0  # the whole mesh, many leaf steps beside short walks
    return mn, mx


def _sorted(r):
    a, f = r.aabb_ids.cpu().numpy(), r.face_ids.cpu().numpy()
    assert np.all(np.diff(a) >= 0)
    return a, f, np.lexsort((f, a))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 4000])
def test_pairs_over_box_counts(orc, n):
    v, f = synthetic.displaced_sphere(3, 8, 0.05, 7)
    mn, mx = _boxes(n, n)
    mesh = MeshBVH(v.cuda(), f.cuda())
    r = mesh.intersect_aabb(torch.from_numpy(mn).cuda(), torch.from_numpy(mx).cuda(), mode=3)
    ref = orc.aabb_pairs(v.numpy(), f.numpy(), mn, mx, mode=3)
    a, fc, o = _sorted(r)
    assert np.array_equal(a[o], ref["aabb_ids"]) and np.array_equal(fc[o], ref["face_ids"])
    assert np.array_equal(r.hit.cpu().numpy(), ref["hit"])
    for k in ("poly_counts", "centroids", "areas", "poly_verts"):
        assert np.array_equal(getattr(r, k).cpu().numpy()[o], ref[k])


def test_kept_and_walked_pairs_in_tree_order(orc):
    v, f = synthetic.displaced_sphere(3, 8, 0.05, 7)
    mn, mx = _boxes(3000, 5)
    mesh = MeshBVH(v.cuda(), f.cuda())
    bmn, bmx = torch.from_numpy(mn).cuda(), torch.from_numpy(mx).cuda()
    r = mesh.intersect_aabb(bmn, bmx, mode=1)
    ref = orc.aabb_pairs(v.numpy(), f.numpy(), mn, mx, mode=1)
    a, fc, o = _sorted(r)
    assert np.array_equal(a[o], ref["aabb_ids"]) and np.array_equal(fc[o], ref["face_ids"])
    counts = np.bincount(a, minlength=len(mn))
    assert (counts == KEPT).any() and (counts == KEPT + 1).any() and (counts > 100).any() and (counts == 0).any()
    # the whole mesh's box lists every face in tree order; so does each box, in part
    place = np.empty(f.shape[0], dtype=np.int64)
    place[fc[a == len(mn) // 2]] = np.arange(f.shape[0])
    same = a[1:] == a[:-1]
    assert np.all(place[fc[1:]][same] > place[fc[:-1]][same])


def test_deep_tree(orc):
    # triangles shrinking by half towards a corner: a tree of one leaf a level
    k = np.arange(96)
    s = np.exp2(-0.5 * k)[:, None, None]
    tri = np.array([[1, 0, 0], [1, 0.4, 0], [1, 0, 0.4]], dtype=np.float64)[None] * s
    v = tri.reshape(-1, 3).astype(np.float32)
    f = np.arange(3 * len(k), dtype=np.int32).reshape(-1, 3)
    mesh = MeshBVH(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda())
    mn = np.full((40, 3), -1.0, dtype=np.float32)
    mx = np.repeat(np.exp2(-np.arange(40))[:, None], 3, axis=1).astype(np.float32) * 1.5
    r = mesh.intersect_aabb(torch.from_numpy(mn).cuda(), torch.from_numpy(mx).cuda(), mode=2)
    ref = orc.aabb_pairs(v, f, mn, mx, mode=2)
    a, fc, o = _sorted(r)
    assert np.array_equal(a[o], ref["aabb_ids"]) and np.array_equal(fc[o], ref["face_ids"])
    assert np.array_equal(r.poly_counts.cpu().numpy()[o], ref["poly_counts"])
