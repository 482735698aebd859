"""The batch autotuner times its samples with the kernel (two or four lanes a
query) and in the order (sorted or the caller's) that the whole call takes."""

import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from atom3d_b200 import synthetic
from atom3d_b200.batch import BatchedMeshBVH, offsets

pytestmark = pytest.mark.gpu


def kernels(fn):
    fn()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    names = {e.name for e in p.events()}
    return ({lanes for lanes in (2, 4) if any(f"udf_group_kernel<{lanes}," in k for k in names)},
            any("batch_query_morton_kernel" in k for k in names))


# samples of 2^16 queries for calls of all three kinds, and the sample sizes that
# fall below the two-lane kernel's and the sort's limits
@pytest.mark.parametrize("queries,sample", [(300_000, 1 << 16), (1_000_000, 1 << 16), (2_200_000, 1 << 21),
                                            (3_000_000, 1 << 21), (2_200_000, 1 << 16)])
def test_samples_run_the_call_s_kernel(queries, sample):
    v, f = synthetic.displaced_sphere(4, 8, 0.05, 1)
    bb = BatchedMeshBVH([(v.cuda(), f.cuda()), (v.cuda() + 4.0, f.cuda())])
    g = torch.Generator(device="cuda").manual_seed(1)
    half = queries // 2
    q = torch.rand(queries, 3, device="cuda", generator=g) * 3 - 1.5
    q[half:] += 4.0
    counts = [half, queries - half]
    qoff = offsets(counts, "cuda")
    call = kernels(lambda: bb.udf(q, counts))
    tune = kernels(lambda: bb.autotune(q, qoff, sample=sample, leaf_sizes=(8,)))
    assert len(call[0]) == 1 and call == tune
    assert bb.tuning.blocks_per_sm >= 1
