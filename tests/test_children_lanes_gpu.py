"""The closest-point kernels' forms by size: four lanes a query or two, in the
caller's order or sorted, with child records or without.  One set of queries on
meshes of slivers, points, flat faces and an infinite vertex, repeated to just
above each change of form, gives the same answers bit for bit in all of them."""

import pytest
import torch

from atom3d_b200.core.mesh_bvh import WideBVH

from test_children_gpu import mesh, plain_query

pytestmark = pytest.mark.gpu

# from here on: two lanes without records, sorting with them, sorting without,
# two lanes with records
SIZES = [(3 << 18) + 3, (7 << 17) + 3, (3 << 19) + 3, (2 << 20) + 3]


@pytest.mark.parametrize("kind", ["soup", "cube", "infinite vertex", "flattened"])
@pytest.mark.parametrize("leaf_max", [1, 8])
def test_every_form_gives_the_same_answers(kind, leaf_max):
    v, f = mesh(kind)
    b = WideBVH(v.cuda(), f.cuda(), leaf_max=leaf_max)
    g = torch.Generator().manual_seed(6)
    fin = v[torch.isfinite(v).all(1)]
    lo, hi = fin.min(0).values, fin.max(0).values
    u = torch.rand(9001, 3, generator=g)
    near = fin[torch.randint(0, fin.shape[0], (3000,), generator=g)]
    near = near + 0.01 * (hi - lo) * torch.randn(3000, 3, generator=g)
    far = (lo + hi) / 2 + (hi - lo).max() * 100 * torch.randn(200, 3, generator=g)
    odd = torch.tensor([[float("nan"), 0, 0], [float("inf"), 0, 0], [0, -float("inf"), 0], [1e30, 0, 0]])
    q = torch.cat([lo + (hi - lo) * (1.4 * u - 0.2), near, far, fin[:300], odd]).contiguous().cuda()
    ref = b.query(q)
    has = ref[1] >= 0  # without a face (NaN or infinite queries) uvw is left unwritten
    for n in SIZES:
        at = torch.arange(n, device="cuda") % q.shape[0]
        big = q[at].contiguous()
        for got in (b.query(big), plain_query(b, big)):
            for x, y in zip((*[r[at] for r in ref[:3]], ref[3][at][has[at]]), (*got[:3], got[3][has[at]])):
                same = (x == y) | ((x != x) & (y != y))
                assert bool(same.all()), (kind, leaf_max, n, int((~same).sum()))
