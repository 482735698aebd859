"""A batch's index guard with child records: a leaf reference outside the
triangle array is recorded in the status and read nowhere, in the four-lane
kernel and in the two-lane one (from 2,097,152 queries on)."""

import pytest
import torch

from atom3d_b200 import _lib, synthetic
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
