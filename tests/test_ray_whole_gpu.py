"""Trees of one node: the pass that takes a whole ray a thread against the
passes that every larger tree takes, all outputs bit for bit.  The same tree is
given to both; only the node count in its view, which chooses, differs."""

import ctypes

import pytest
import torch

from atom3d_b200 import MeshBVH, _lib

pytestmark = pytest.mark.gpu


def _nearest(mesh, view, o, d, max_t, optional):
    n = o.shape[0]
    ws = _lib.workspace(_lib.lib().a3d_ray_workspace_bytes(n), o.device)
    out = [torch.full(s, 7, dtype=t, device="cuda") for s, t in
           (((n,), torch.uint8), ((n,), torch.float32), ((n,), torch.int32), ((n, 3), torch.float32),
            ((n, 3), torch.float32), ((n, 3), torch.float32))]
    rest = [x.data_ptr() if optional else None for x in out[3:]]
    _lib.call("a3d_ray_nearest", ctypes.byref(view), o.data_ptr(), d.data_ptr(), n, max_t,
              mesh.get_face_normals().data_ptr() if optional else None, *[x.data_ptr() for x in out[:3]], *rest,
              ws.data_ptr(), ws.numel(), _lib.stream_ptr(o.device))
    status = (ctypes.c_uint32 * 2)()
    _lib.call("a3d_ray_status", ws.data_ptr(), status, _lib.stream_ptr(o.device))
    assert list(status) == [0, 0]
    return out


@pytest.mark.parametrize("tris", [1, 2, 8, 9, 20])
@pytest.mark.parametrize("n", [1, 127, 129, 5003])
@pytest.mark.parametrize("max_t", [1e10, 0.7, 0.0, -1.0, float("inf"), float("nan")])
@pytest.mark.parametrize("optional", [True, False])
def test_whole_rays_against_the_general_passes(tris, n, max_t, optional):
    g = torch.Generator().manual_seed(100 * tris + n)
    v = (torch.rand(tris, 1, 3, generator=g) - 0.5 + 0.6 * torch.randn(tris, 3, 3, generator=g)).reshape(-1, 3)
    mesh = MeshBVH(v.cuda(), torch.arange(3 * tris, dtype=torch.int32).reshape(-1, 3).cuda())
    view = mesh._bvh.view
    if view.num_nodes != 1:
        assert tris > 8
        pytest.skip("the builder made more than one node of these triangles")
    o = torch.randn(n, 3, generator=g)
    d = torch.randn(n, 3, generator=g)
    d[::5] = torch.eye(3)[torch.randint(0, 3, (len(d[::5]),), generator=g)]  # along an axis
    k = min(n, tris)  # at a vertex, and from one
    d[:k] = v[: 3 * k : 3] - o[:k]
    o[n // 2 : n // 2 + 1] = v[0]
    if n > 100:
        o[20], d[21], d[22] = float("nan"), float("inf"), 0.0
        o[23] = 1e30
    o, d = o.cuda(), d.cuda()
    general = _lib.BvhView.from_buffer_copy(view)
    general.num_nodes = 2
    for a, b in zip(_nearest(mesh, view, o, d, max_t, optional), _nearest(mesh, general, o, d, max_t, optional)):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
