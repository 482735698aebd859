"""Flood fill labels either side of the volume size from which tiles are longer
(2^18 words), and with each length of the rows' runs, against the oracle's
breadth-first fill; lists in their order."""

import numpy as np
import pytest
import torch

from atom3d_b200 import flood_fill_3d_sparse

pytestmark = pytest.mark.gpu


# volumes of dims + 4: 258,048 and 262,144 words (runs of 4 rows), 500,000 (8), 1,351,680 (16)
@pytest.mark.parametrize("dims,conn", [((59, 124, 1020), 18), ((60, 124, 1020), 26), ((246, 246, 250), 6),
                                       ((252, 348, 476), 26)])
@pytest.mark.parametrize("density", [0.03, 0.6])
def test_labels_match_oracle(orc, dims, conn, density):
    g = np.random.default_rng([dims[0], int(100 * density)])
    m = g.random(dims) < density
    m[0, 0, 0] = m[tuple(d - 1 for d in dims)] = True
    dam = np.argwhere(m).astype(np.int64) + 2
    got = flood_fill_3d_sparse(torch.from_numpy(dam).cuda(), 1024, padding=2, connectivity=conn)
    ref = orc.flood_fill_3d_sparse(dam, 1024, padding=2, connectivity=conn)
    for a, b, name in zip(got, ref, ["water", "dry", "tide", "dam", "dam_mask", "ext"]):
        a = a.cpu().numpy()
        assert a.shape == b.shape and np.array_equal(a, b), (name, a.shape, b.shape)
