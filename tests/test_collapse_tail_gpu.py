"""Trees that outlast the collapse's grid launches, so that its last block
collapses levels of hundreds of nodes: triangles over many octaves of size in
one mesh, and the same mesh in a batch of more meshes than the first block
takes."""

import numpy as np
import pytest
import torch

from atom3d_b200 import MeshBVH
from atom3d_b200.batch import BatchedMeshBVH
from atom3d_b200.core.mesh_bvh import WideBVH

from test_collapse_gpu import _check

pytestmark = pytest.mark.gpu

HEAD_NODES, GRID_LEVELS = 256, 12


def octaves(n, span):
    g = np.random.default_rng(n)
    s = np.exp2(-span * g.random((n, 1, 1)))
    return torch.from_numpy((s * (1 + g.random((n, 3, 3)))).reshape(-1, 3).astype(np.float32))


def level_sizes(nodes, roots):
    w = nodes.cpu().numpy().view(np.uint32).reshape(-1, 16)
    level, sizes = np.asarray(roots, dtype=np.int64), []
    while level.size:
        sizes.append(level.size)
        ref, used = w[level, 10:14], np.arange(4)[None] < (w[level, 3] >> 24)[:, None]
        level = ref[used & (ref >> 31 == 0)].astype(np.int64)
    return sizes


def tail(sizes, head_nodes=HEAD_NODES):
    first = next((i for i, k in enumerate(sizes) if k > head_nodes), len(sizes))
    return sizes[first + GRID_LEVELS:]


def test_one_mesh():
    v = octaves(100_000, 20)
    f = torch.arange(v.shape[0], dtype=torch.int32).reshape(-1, 3)
    b = WideBVH(v.cuda(), f.cuda())
    assert max(tail(level_sizes(b.nodes, [0]))) > 256
    _check(v)


def test_many_meshes():
    deep = octaves(20_000, 20).cuda()
    small = octaves(5, 1).cuda()
    face = lambda v: torch.arange(v.shape[0], dtype=torch.int32, device="cuda").reshape(-1, 3)  # noqa: E731
    meshes = [(small, face(small))] * HEAD_NODES + [(deep, face(deep))]
    bb = BatchedMeshBVH(meshes)
    n = int(bb.num_nodes.item())
    sizes = level_sizes(bb.nodes[:n * 64], bb.roots.tolist())
    assert sizes[0] == HEAD_NODES + 1 and sum(sizes) == n and len(tail(sizes)) > 5
    g = torch.Generator(device="cuda").manual_seed(2)
    q = torch.rand(20_000, 3, device="cuda", generator=g) ** 6 * 2  # down to the small triangles
    got = bb.udf(q, [0] * HEAD_NODES + [q.shape[0]])
    ref = MeshBVH(deep, face(deep)).udf(q, return_closest=True)
    assert torch.equal(got[0], ref.distances)
    q1 = torch.rand(HEAD_NODES * 8, 3, device="cuda", generator=g)
    got = bb.udf(q1, [8] * HEAD_NODES + [0])
    assert torch.equal(got[0], MeshBVH(small, face(small)).udf(q1))
