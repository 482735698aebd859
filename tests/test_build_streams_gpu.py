"""A constructed tree is finished: a query on another stream right after the
constructor, without any wait, reads the whole tree and its child records, also
when the records did not fit the capacity guessed before the build."""

import pytest
import torch

from atom3d_b200 import synthetic
from atom3d_b200.core.mesh_bvh import WideBVH

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf_max,capacity", [(8, None), (1, None), (8, 1)])
def test_query_on_another_stream_after_the_build(monkeypatch, leaf_max, capacity):
    if capacity is not None:
        monkeypatch.setattr(WideBVH, "_child_capacity", staticmethod(lambda nf, lm: capacity))
    v, f = synthetic.displaced_sphere(6, 8, 0.05, 1)
    v, f = v.cuda(), f.cuda()
    q = torch.rand(4000, 3, generator=torch.Generator().manual_seed(3)).cuda() * 3 - 1.5
    build, query = torch.cuda.Stream(), torch.cuda.Stream()
    ref = WideBVH(v, f, leaf_max=leaf_max).query(q)
    torch.cuda.synchronize()
    for _ in range(50):
        with torch.cuda.stream(build):
            b = WideBVH(v, f, leaf_max=leaf_max)
        with torch.cuda.stream(query):
            got = b.query(q)
        torch.cuda.synchronize()
        for x, y in zip(ref, got):
            assert torch.equal(x, y)


@pytest.mark.parametrize("leaf_max", [1, 3, 8])
def test_the_guessed_capacity_holds_usual_trees(leaf_max):
    for level in (1, 4, 6):
        v, f = synthetic.displaced_sphere(level, 8, 0.05, 1)
        b = WideBVH(v.cuda(), f.cuda(), leaf_max=leaf_max)
        assert b.num_nodes <= WideBVH._child_capacity(f.shape[0], leaf_max)
