"""The collapse into wide nodes where its launches change: builds that one block
collapses alone, the first sizes beyond, and skewed trees that outlast the
levels run by the grid.  Every triangle lies in exactly one leaf, inside every
box above it, and nodes come in breadth-first order."""

import numpy as np
import pytest
import torch

from atom3d_b200.core.mesh_bvh import WideBVH

pytestmark = pytest.mark.gpu


def _soup(n):
    g = torch.Generator().manual_seed(n)
    v = torch.rand(n, 1, 3, generator=g) + 0.05 * torch.rand(n, 3, 3, generator=g)
    return v.reshape(-1, 3).float()


def _skewed(n):
    # a chain of triangles halving towards the origin (each split cuts a few
    # off), and the rest at its start
    k = np.arange(n)
    s = np.where(k < 220, np.exp2(-0.5 * np.minimum(k, 220)), 1.0)[:, None, None]
    tri = np.array([[1, 0, 0], [1, 0.4, 0], [1, 0, 0.4]], dtype=np.float64)[None] * s
    rest = np.random.default_rng(n).uniform(0, 0.01, (n, 1, 3)) * (k >= 220)[:, None, None]
    return torch.from_numpy((tri + rest).reshape(-1, 3).astype(np.float32))


def _check(v):
    n = v.shape[0] // 3
    b = WideBVH(v.cuda(), torch.arange(3 * n, dtype=torch.int32).reshape(-1, 3).cuda())
    w = b.nodes.cpu().numpy().view(np.uint32).reshape(-1, 16)
    f = w.view(np.float32)
    t = b.tris.cpu().numpy().view(np.float32).reshape(-1, 16)
    tv = np.stack([t[:, 0:3], t[:, 4:7], t[:, 8:11]], 1)
    face = np.sort(b.tris.cpu().numpy().view(np.int32).reshape(-1, 16)[:, 3])
    assert np.array_equal(face, np.arange(n))
    byte = (w[:, 4:10, None] >> (8 * np.arange(4, dtype=np.uint32))) & 255
    scale = np.stack([((w[:, 3] >> (8 * a)) & 255) << 23 for a in range(3)], 1).astype(np.uint32).view(np.float32)
    # origin + q * scale, rounded once to FP32 as the traversals do (the product is exact)
    lo = f[:, 0:3, None] + (byte[:, 0:3] * scale[:, :, None]).astype(np.float32)
    hi = f[:, 0:3, None] + (byte[:, 3:6] * scale[:, :, None]).astype(np.float32)
    seen = np.zeros(n, dtype=np.int64)
    visited = np.zeros(w.shape[0], dtype=np.int64)
    stack = [(0, np.full(3, -np.inf), np.full(3, np.inf), 0)]
    depth = 0
    order = []
    while stack:
        i, l0, h0, d = stack.pop()
        visited[i] += 1
        order.append((d, i))
        depth = max(depth, d)
        for c in range(int(w[i, 3] >> 24)):
            r = int(w[i, 10 + c])
            l1, h1 = np.maximum(l0, lo[i, :, c]), np.minimum(h0, hi[i, :, c])
            if r & 0x80000000:
                first, cnt = r & 0x0FFFFFFF, ((r >> 28) & 7) + 1
                seen[first:first + cnt] += 1
                p = tv[first:first + cnt].reshape(-1, 3)
                assert (p >= l1).all() and (p <= h1).all()
            else:
                stack.append((r, l1, h1, d + 1))
    assert (seen == 1).all() and (visited == 1).all()
    levels = [d for d, _ in sorted(order, key=lambda e: e[1])]
    assert levels == sorted(levels)  # breadth first
    return depth


@pytest.mark.parametrize("n", [1, 2, 9, 255, 2047, 2048, 2049, 2500, 20000])
def test_even_trees(n):
    _check(_soup(n))


@pytest.mark.parametrize("n", [200, 2048, 2049, 6000])
def test_skewed_trees(n):
    assert _check(_skewed(n)) >= 8
