"""A batch's index guard with child records: a leaf reference outside the
triangle array is recorded in the status and read nowhere, in the four-lane
kernel and in the two-lane one (from 2,097,152 queries on)."""

import pytest
import torch

from atom3d_b200 import MeshBVH, _lib, synthetic
from atom3d_b200.batch import BatchedMeshBVH

pytestmark = pytest.mark.gpu

FAULT_TRI = 2
LEAF = -0x80000000  # bit 31 of an int32


@pytest.mark.parametrize("queries", [3000, (2 << 20) + 5])
def test_leaf_outside_the_arrays_is_recorded(queries):
    v, f = synthetic.displaced_sphere(3, 8, 0.05, 1)
    bb = BatchedMeshBVH([(v.cuda(), f.cuda()), (v.cuda() + 4.0, f.cuda())])
    ref = bb.nodes[:int(bb.num_nodes.item()) * 64].view(torch.int32).view(-1, 16)[:, 10:14]
    leaves = torch.nonzero((ref < 0) & (ref != -1))
    for node, c in leaves[::7].tolist():
        ref[node, c] = LEAF | 0x0FFFFF00  # one triangle, far past the end
    _lib.call("a3d_bvh_children", bb.nodes.data_ptr(), bb.tris.data_ptr(), bb.num_children, bb.num_nodes.data_ptr(),
              bb.num_faces, bb.children.data_ptr(), _lib.stream_ptr(bb.device))
    g = torch.Generator(device="cuda").manual_seed(1)
    half = queries // 2
    q = torch.rand(queries, 3, device="cuda", generator=g) * 3 - 1.5
    q[half:] += 4.0
    bb.udf(q, [half, queries - half])
    assert bb.query_status()["faults"] == FAULT_TRI


def test_tree_above_the_level_limit_is_reported_and_safe():
    """Triangles over 100 octaves make a tree deeper than the collapse's level
    limit.  The build's status says so; a query without reading it stays inside
    the arrays, says so too, and answers for the other mesh of the batch."""
    g = torch.Generator().manual_seed(4)
    s = torch.exp2(-100 * torch.rand(60_000, 1, 1, generator=g, dtype=torch.float64))
    deep = (s * (1 + torch.rand(60_000, 3, 3, generator=g, dtype=torch.float64))).reshape(-1, 3).float().cuda()
    v, f = synthetic.displaced_sphere(3, 8, 0.05, 1)
    meshes = [(deep, torch.arange(180_000, dtype=torch.int32).reshape(-1, 3).cuda()), (v.cuda(), f.cuda())]
    bb = BatchedMeshBVH(meshes, build=False)
    bb.build()
    with pytest.raises(RuntimeError):
        bb.check()
    q = torch.zeros(6000, 3, device="cuda")
    q[:3000] = torch.exp2(-140 * torch.rand(3000, 1, generator=g)).cuda()
    q[3000:] = torch.rand(3000, 3, generator=g).cuda() * 3 - 1.5
    dist, _, _ = bb.udf(q, [3000, 3000])
    assert bb.query_status()["faults"] == FAULT_TRI
    assert torch.equal(dist[3000:], MeshBVH(v.cuda(), f.cuda()).udf(q[3000:]))
