"""The child records only skip work: a3d_udf_children returns what a3d_udf
(no records) returns, bit for bit, because a child is skipped only when none of its
triangles' computed distances can be below the best one."""

import ctypes

import pytest
import torch

from atom3d_b200 import _lib, synthetic
from atom3d_b200.core.mesh_bvh import WideBVH

pytestmark = pytest.mark.gpu


def plain_query(b, p):
    n = p.shape[0]
    d = torch.empty(n, device="cuda")
    f = torch.empty(n, dtype=torch.int32, device="cuda")
    cp = torch.empty(n, 3, device="cuda")
    uvw = torch.empty(n, 3, device="cuda")
    ws = _lib.workspace(_lib.lib().a3d_udf_workspace_bytes(n, 1), p.device)
    _lib.call("a3d_udf", ctypes.byref(b.view), p.data_ptr(), n, d.data_ptr(), f.data_ptr(), cp.data_ptr(),
              uvw.data_ptr(), None, None, None, 1, ws.data_ptr(), ws.numel(), _lib.stream_ptr(p.device))
    return d, f, cp, uvw


def box_mesh(k):
    """Axis-aligned cube surface, k x k quads a face: box, plane and triangle
    distances coincide exactly."""
    r = torch.arange(k + 1, dtype=torch.float32) / k * 2 - 1
    v, f = [], []
    for a in range(3):
        for s in (-1.0, 1.0):
            g = torch.stack(torch.meshgrid(r, r, indexing="ij"), -1).reshape(-1, 2)
            p = torch.empty(g.shape[0], 3)
            p[:, a], p[:, (a + 1) % 3], p[:, (a + 2) % 3] = s, g[:, 0], g[:, 1]
            i = torch.arange(k)[:, None] * (k + 1) + torch.arange(k)[None]
            i = i.reshape(-1) + len(v) * (k + 1) ** 2
            f += [torch.stack([i, i + 1, i + k + 2], 1), torch.stack([i, i + k + 2, i + k + 1], 1)]
            v.append(p)
    return torch.cat(v), torch.cat(f).int()


def mesh(kind):
    g = torch.Generator().manual_seed(11)
    if kind == "one triangle":
        return torch.rand(3, 3, generator=g), torch.tensor([[0, 1, 2]], dtype=torch.int32)
    if kind == "cube":
        return box_mesh(9)
    if kind == "soup":  # random triangles of every size, slivers and points among them
        v = torch.rand(3000, 3, generator=g)
        v[1:900:3] = v[0:900:3] + 0.01 * torch.randn(300, 3, generator=g)
        v[2:900:3] = v[0:900:3] + torch.tensor([1e-7, 0.2, 0.1])
        v[1500:1530] = v[1500]
        return v, torch.arange(3000, dtype=torch.int32).reshape(-1, 3)
    if kind == "infinite vertex":
        v, f = synthetic.displaced_sphere(3, 8, 0.05, 2)
        v = v.clone()
        v[7, 1] = float("inf")
        return v, f
    v, f = synthetic.displaced_sphere(5, 16, 0.05, 3)
    if kind == "far from the origin":
        v = v + torch.tensor([3000.0, -40.0, 7.0])
    if kind == "flattened":
        v = v * torch.tensor([1.0, 1e-3, 2.0])
    return v, f


@pytest.mark.parametrize("kind", ["smooth", "one triangle", "cube", "soup", "infinite vertex", "far from the origin",
                                  "flattened"])
@pytest.mark.parametrize("leaf_max", [1, 8])
def test_child_records_change_no_result(kind, leaf_max):
    v, f = mesh(kind)
    b = WideBVH(v.cuda(), f.cuda(), leaf_max=leaf_max)
    g = torch.Generator().manual_seed(5)
    fin = v[torch.isfinite(v).all(1)]
    lo, hi = fin.min(0).values, fin.max(0).values
    u = torch.rand(20011, 3, generator=g)
    near = fin[torch.randint(0, fin.shape[0], (5000,), generator=g)]
    near = near + 0.01 * (hi - lo) * torch.randn(5000, 3, generator=g)
    far = (lo + hi) / 2 + (hi - lo).max() * 100 * torch.randn(500, 3, generator=g)
    centre = ((lo + hi) / 2).expand(50, 3)
    odd = torch.tensor([[float("nan"), 0, 0], [float("inf"), 0, 0], [0, -float("inf"), 0], [1e30, 0, 0]])
    for q in (torch.cat([lo + (hi - lo) * (1.4 * u - 0.2), near, far, centre, fin[:300], odd]), centre[:1]):
        q = q.contiguous().cuda()
        ref, got = plain_query(b, q), b.query(q)
        has = ref[1] >= 0  # without a face (NaN or infinite queries) uvw is left unwritten
        for x, y in zip((*ref[:3], ref[3][has]), (*got[:3], got[3][has])):
            same = (x == y) | ((x != x) & (y != y))
            assert bool(same.all()), (kind, leaf_max, int((~same).sum()))


@pytest.mark.parametrize("kind", ["one triangle", "cube"])
def test_flat_boxes_still_give_every_query_its_face(kind):
    """A flat box can round to just beyond its own triangle: a query whose
    radius that triangle seeds must not come back empty."""
    v, f = mesh(kind)
    if kind == "one triangle":
        v = torch.tensor([[0.0, 0, 0], [1, 0, 0], [0, 1, 0]])
    b = WideBVH(v.cuda(), f.cuda())
    q = torch.rand(50000, 3, generator=torch.Generator().manual_seed(2)).cuda() * 3 - 1
    first = b.query(q)
    assert int(first[1].min()) >= 0
    for _ in range(3):
        for x, y in zip(first, b.query(q)):
            assert torch.equal(x, y)


@pytest.mark.parametrize("leaf_max", [1, 8])
@pytest.mark.parametrize("bounded", [False, True])
def test_greedy_seed_ends_where_no_box_distance_is_finite(leaf_max, bounded):
    """The greedy descent for a seed (NO_REUSE) on queries whose squared box
    distances overflow or are NaN: the answer of the default seeding."""
    v, f = mesh("smooth")
    b = WideBVH(v.cuda(), f.cuda(), leaf_max=leaf_max)
    inf, nan = float("inf"), float("nan")
    odd = torch.tensor([[inf, 0, 0], [0, -inf, 0], [inf, inf, -inf], [1e30, 0, 0], [0, 2e19, -3e19], [3e38, 3e38, 3e38],
                        [nan, 0, 0], [nan, nan, inf]])
    g = torch.Generator().manual_seed(8)
    q = torch.cat([odd, torch.rand(300, 3, generator=g) * 3 - 1.5, odd, odd[:1].expand(40, 3)]).contiguous().cuda()
    ref = b.query(q)
    seeding, bound = _lib.A3D_UDF_NO_REUSE, None
    if bounded:
        seeding |= _lib.A3D_UDF_BOUND_SEEDS
        bound = torch.full((q.shape[0],), inf, device="cuda")
        bound[::2] = 10.0
    got = b.query(q, bound=bound, seeding=seeding)
    has = ref[1] >= 0
    assert not bool(has[:8].any()) and bool(has[8:308].all())
    for x, y in zip((*ref[:3], ref[3][has]), (*got[:3], got[3][has])):
        assert bool(((x == y) | ((x != x) & (y != y))).all())
