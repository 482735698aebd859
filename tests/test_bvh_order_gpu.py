"""The leaf order of the SAH build on meshes whose nodes meet every way of
splitting them (one triangle a lane, a warp's bins, a block's bins), against
orders recorded from the builder that split every small node with a warp's
bins (golden/bvh_order.npz)."""

import os

import numpy as np
import pytest
import torch

from atom3d_b200.core.mesh_bvh import WideBVH

pytestmark = pytest.mark.gpu

SIZES = (2, 3, 31, 32, 33, 65, 255, 256, 257, 513, 1500, 2600)
GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "bvh_order.npz")


def soup(n):
    """n random triangles of mixed size, an eighth of them one and the same
    place (no split between them) and an eighth in one plane."""
    g = torch.Generator().manual_seed(n)
    c = torch.rand(n, 1, 3, generator=g)
    v = c + 0.3 * torch.rand(n, 3, 3, generator=g) * torch.rand(n, 1, 1, generator=g)
    k = n // 8
    v[:k] = v[:1]
    v[k:2 * k, :, 1] = 0.25
    return v.reshape(-1, 3), torch.arange(3 * n, dtype=torch.int32).reshape(-1, 3)


def leaf_order(n):
    v, f = soup(n)
    b = WideBVH(v.cuda(), f.cuda())
    return b.tris.view(torch.int32).view(-1, 16)[:, 3].cpu().numpy()  # face ids in leaf order


@pytest.mark.parametrize("n", SIZES)
def test_leaf_order_is_unchanged(n):
    assert np.array_equal(leaf_order(n), np.load(GOLDEN)[f"n{n}"])
