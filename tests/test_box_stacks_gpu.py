"""The pair walk of MeshBVH.intersect_aabb where a box's stack outgrows shared
memory.  Against the oracle's brute force; within a box the faces come in tree
order."""

import numpy as np
import pytest
import torch

from atom3d_b200 import MeshBVH

pytestmark = pytest.mark.gpu

SHARED = 32  # stack entries of a box in shared memory


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


def _deepest_stack(mesh):
    """Entries on the stack of a walk that meets every child."""
    words = mesh._bvh.nodes.view(torch.int32).view(-1, 16).cpu().numpy().view(np.uint32)
    stack, deepest = [0], 0
    while stack:
        ref = stack.pop()
        if not ref >> 31:
            node = words[ref]
            stack += [int(x) for x in node[10 : 10 + (int(node[3]) >> 24)][::-1]]
            deepest = max(deepest, len(stack) - 1)
    return deepest


@pytest.mark.parametrize("n", [1, 31, 4500])
def test_stacks_beyond_shared_memory(orc, n):
    # overlapping triangles that shrink towards a corner: a deep, skewed tree
    g = np.random.default_rng(11)
    t = 6000
    s = (0.997 ** np.arange(t))[:, None, None]
    v = (s * (np.array([1.0, 0.3, 0.1]) + 0.3 * g.normal(size=(t, 3, 3)))).astype(np.float32).reshape(-1, 3)
    f = np.arange(3 * t, dtype=np.int32).reshape(-1, 3)
    mesh = MeshBVH(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda())
    assert _deepest_stack(mesh) > SHARED
    c = v[g.integers(0, len(v), n)]
    h = np.exp(g.uniform(np.log(1e-4), np.log(0.02), (n, 1)))
    mn, mx = (c - h).astype(np.float32), (c + h).astype(np.float32)
    mn[::500], mx[::500] = -9.0, 9.0  # every triangle
    counts = _check(orc, mesh, v, f, mn, mx)
    assert np.all(counts[::500] == t)
