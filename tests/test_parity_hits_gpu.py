"""Parity votes of rays with as many hits as shared memory holds, one more, up to
the 256 a ray keeps, and of rays whose stack outgrows shared memory; votes equal
to the oracle's brute force."""

import ctypes

import numpy as np
import pytest
import torch

from atom3d_b200 import MeshBVH, _lib

pytestmark = pytest.mark.gpu

KEPT = 256  # hits a ray keeps


def votes_of(v, f, p, dirs, coalesce=1e-4):
    mesh = MeshBVH(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda())
    pts, d = torch.from_numpy(p).cuda(), torch.from_numpy(dirs).cuda()
    votes = torch.empty(len(p), dtype=torch.int32, device="cuda")
    ws = _lib.workspace(_lib.lib().a3d_ray_workspace_bytes(0), pts.device)
    _lib.call("a3d_ray_parity_votes", ctypes.byref(mesh._bvh.view), pts.data_ptr(), len(p), d.data_ptr(), len(dirs), 1e6,
              coalesce, votes.data_ptr(), ws.data_ptr(), ws.numel(), _lib.stream_ptr(pts.device))
    st = (ctypes.c_uint32 * 2)()
    _lib.call("a3d_ray_status", ws.data_ptr(), st, _lib.stream_ptr(pts.device))
    return votes.cpu().numpy(), bool(st[1])


def sheets(z, g):
    """A triangle across every height z, either way up, in any order."""
    z = g.permutation(z)
    t = np.array([[-900.0, -800, 0], [1000, -700, 0], [50, 1200, 0]])[None].repeat(len(z), 0)
    t[:, :, 2] = z[:, None]
    flip = g.random(len(z)) < 0.5
    t[flip] = t[flip][:, ::-1]
    return t.reshape(-1, 3).astype(np.float32), np.arange(3 * len(z), dtype=np.int32).reshape(-1, 3)


DIRS = np.array([[0.03, -0.02, 1], [-0.05, 0.04, 1], [0.01, 0.02, 1]], dtype=np.float32)


@pytest.mark.parametrize("hits", [1, 11, 12, 13, 31, 32, 33, 63, 64, 65, 255, 256])
@pytest.mark.parametrize("n", [1, 40, 3001])
def test_hits_up_to_the_kept_ones(orc, hits, n):
    g = np.random.default_rng([hits, n])
    z = np.arange(1.0, hits + 1)
    z[1::5] = z[0::5][:len(z[1::5])] + 5e-5  # merged with the sheet below
    v, f = sheets(z, g)
    p = np.zeros((n, 3), dtype=np.float32)
    p[:, :2] = g.uniform(-20, 20, (n, 2))
    p[n // 2:, 2] = g.uniform(0, hits + 1, n - n // 2)  # some rays start among the sheets
    got, lost = votes_of(v, f, p, DIRS)
    assert not lost
    assert np.array_equal(got, orc.parity_votes(v, f, p, DIRS))


def test_more_hits_than_kept_are_reported():
    v, f = sheets(np.arange(1.0, KEPT + 2), np.random.default_rng(1))
    p = np.zeros((70, 3), dtype=np.float32)
    assert votes_of(v, f, p, DIRS)[1]
    p[:, 2] = 1.5
    assert not votes_of(v, f, p, DIRS)[1]


def test_stacks_beyond_shared_memory(orc):
    """Needles across the whole volume: a ray meets most boxes of the tree and
    few triangles."""
    g = np.random.default_rng(5)
    a = g.uniform(-1, 1, (20000, 1, 3))
    b = -a + 0.2 * g.normal(size=(20000, 1, 3))
    t = np.concatenate([a, b, b + 2e-3 * g.normal(size=(20000, 1, 3))], 1)
    v, f = t.reshape(-1, 3).astype(np.float32), np.arange(60000, dtype=np.int32).reshape(-1, 3)
    p = g.uniform(-1.2, 1.2, (300, 3)).astype(np.float32)
    d = g.normal(size=(4, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    got, lost = votes_of(v, f, p, d)
    assert not lost
    assert np.array_equal(got, orc.parity_votes(v, f, p, d))
