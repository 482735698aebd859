"""Rays without an end: max_t = inf (or so large that the pruning limit
overflows) gives the hits of a large finite max_t, nearest, all and by parity;
empty slots of the tree are not entered."""

import math

import pytest
import torch

from atom3d_b200 import MeshBVH, synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[1, 5, 20480])
def rays(request):
    v, f = synthetic.displaced_sphere(5, 8, 0.1, 1)
    mesh = MeshBVH(v.cuda(), f[:request.param].contiguous().cuda())
    g = torch.Generator().manual_seed(1)
    o = torch.rand(5000, 3, generator=g) * 3 - 1.5
    d = torch.nn.functional.normalize(torch.randn(5000, 3, generator=g), dim=1)
    return mesh, o.cuda(), d.cuda()


@pytest.mark.parametrize("max_t", [math.inf, 3.4028234e38])
def test_unbounded_rays(rays, max_t):
    mesh, o, d = rays
    ref, got = mesh.intersect_ray(o, d, max_t=1e30), mesh.intersect_ray(o, d, max_t=max_t)
    assert torch.equal(ref.hit, got.hit) and torch.equal(ref.face_ids, got.face_ids)
    assert torch.equal(ref.t[ref.hit], got.t[ref.hit]) and bool((got.t[~ref.hit] == max_t).all())
    assert torch.equal(ref.hit_points, got.hit_points)
    ra, ga = (mesh.intersect_ray(o, d, max_t=t, mode="all") for t in (1e30, max_t))
    for name in ("ray_idx", "t", "face_ids", "sign", "hit_points"):
        assert torch.equal(getattr(ra, name), getattr(ga, name)), name
    assert torch.equal(mesh.sdf(o, mode="parity", max_t=1e30), mesh.sdf(o, mode="parity", max_t=max_t))
    assert mesh.ray_status()["overflow"] == 0
