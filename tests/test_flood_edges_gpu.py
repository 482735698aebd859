"""Flood fill labels at the edges of the brick, row and word blocking: random
dams (scattered, tangled near the percolation threshold of 6-connectivity, and
dense) in boxes that no block size divides, for each connectivity, against the
oracle's breadth-first fill; lists in their order."""

import numpy as np
import pytest
import torch

from atom3d_b200 import flood_fill_3d_sparse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conn", [6, 18, 26])
@pytest.mark.parametrize("dims,res", [((1, 1, 1), 8), ((31, 33, 95), 256), ((70, 47, 131), 256), ((9, 35, 1100), 2048)])
@pytest.mark.parametrize("density", [0.02, 0.35, 0.8])
def test_random_dams_match_oracle(orc, conn, dims, res, density):
    g = np.random.default_rng(hash((conn, dims, density)) % 2 ** 32)
    m = g.random(dims) < density
    m[tuple(d // 2 for d in dims)] = True
    lo = g.integers(1, 4, 3)
    dam = (np.argwhere(m) + lo).astype(np.int64)
    got = flood_fill_3d_sparse(torch.from_numpy(dam).cuda(), res, padding=2, connectivity=conn)
    ref = orc.flood_fill_3d_sparse(dam, res, padding=2, connectivity=conn)
    for a, b, name in zip(got, ref, ["water", "dry", "tide", "dam", "dam_mask", "ext"]):
        a = a.cpu().numpy()
        assert a.shape == b.shape and np.array_equal(a, b), (name, a.shape, b.shape)
