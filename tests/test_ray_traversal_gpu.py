"""The persistent ray kernels where their buffers end: few rays, partial
warps, rays whose stack or hit buffer outgrows shared memory."""

import pytest
import torch

from atom3d_b200 import MeshBVH, synthetic

pytestmark = pytest.mark.gpu


def shells(k):
    """k concentric spheres of radius 1, 2, ... k."""
    v, f = synthetic.icosphere(2)
    vs = torch.cat([v * (i + 1) for i in range(k)])
    fs = torch.cat([f + i * v.shape[0] for i in range(k)])
    return vs, fs


@pytest.mark.parametrize("n", [1, 31, 33, 129, 20000])
@pytest.mark.parametrize("kind", ["soup", "shells"])
def test_nearest_is_the_first_of_all_hits(kind, n):
    g = torch.Generator().manual_seed(n)
    if kind == "soup":  # overlapping triangles: many boxes at once on a ray's stack
        v = torch.rand(20000, 1, 3, generator=g) + 0.4 * torch.randn(20000, 3, 3, generator=g)
        v, f = v.reshape(-1, 3), torch.arange(60000, dtype=torch.int32).reshape(-1, 3)
        o = torch.rand(n, 3, generator=g) * 4 - 2
    else:
        v, f = shells(20)
        o = torch.rand(n, 3, generator=g) * 50 - 25
    d = torch.randn(n, 3, generator=g)
    d = d / d.norm(dim=1, keepdim=True)
    mesh = MeshBVH(v.cuda(), f.cuda())
    o, d = o.cuda(), d.cuda()
    near = mesh.intersect_ray(o, d)
    assert mesh.ray_status()["overflow"] == 0
    every = mesh.intersect_ray(o, d, mode="all")
    first = torch.full((n,), 1e10, device="cuda").scatter_reduce(0, every.ray_idx.long(), every.t, "amin")
    # "all" leaves out grazing hits, so the nearest one may come earlier, never later
    assert bool((near.t <= first).all())
    grazing = near.t < first
    nd = (near.normals * d).sum(1).abs()
    assert bool((nd[grazing] < 2e-4).all())
    assert torch.equal(near.hit, near.t < 1e10) and torch.equal(near.hit, near.face_ids >= 0)
    p = o + near.t[:, None] * d
    assert torch.allclose(near.hit_points[near.hit], p[near.hit], atol=1e-5)


@pytest.mark.parametrize("n", [1, 33, 3000])
def test_parity_through_many_shells(n):
    """Points among 40 shells: their rays cross up to 40 of them, past the hits
    kept in shared memory.  Against the crossings the all-hits query counts
    (its rays in other directions; a ray through an edge may count one twice,
    so the majority of directions decides on both sides)."""
    k = 40
    v, f = shells(k)
    g = torch.Generator().manual_seed(n)
    j = torch.randint(0, k, (n,), generator=g)
    r = j + 0.2 + 0.5 * torch.rand(n, generator=g)
    p = torch.randn(n, 3, generator=g)
    p = (p / p.norm(dim=1, keepdim=True) * r[:, None]).cuda()
    mesh = MeshBVH(v.cuda(), f.cuda())
    sdf = mesh.sdf(p, mode="parity")
    assert mesh.ray_status()["overflow"] == 0
    odd = torch.zeros(n, device="cuda")
    for _ in range(9):
        d = torch.randn(1, 3, generator=g)
        d = (d / d.norm()).cuda().expand(n, 3).contiguous()
        hits = mesh.intersect_ray(p, d, mode="all")
        odd += torch.bincount(hits.ray_idx.long(), minlength=n) % 2
    assert torch.equal(sdf < 0, odd > 4)
