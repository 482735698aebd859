"""Workspaces sized for a number of queries or keys serve every smaller call:
the sizes asked for never fall as the number grows."""

import pytest

from atom3d_b200.batch import _bind


def sizes():
    edges = [512, 65536, 131072, 303104, 606208, 786432, 917504, 1048576, 1212416, 1572864, 2097152, 8388608, 16777216]
    n = {1, 2, 3}
    for e in edges:
        n |= set(range(e - 40, e + 41, 5)) | {e - 1, e, e + 1} | {int(e * k / 16) for k in range(17, 32)}
    return sorted(n)


@pytest.mark.parametrize("name", ["udf sorted", "udf unsorted", "batch", "sort", "batch autotune"])
def test_sizes_never_fall(lib, name):
    bind = _bind()
    size = {
        "udf sorted": lambda n: lib.a3d_udf_workspace_bytes(n, 1),
        "udf unsorted": lambda n: lib.a3d_udf_workspace_bytes(n, 0),
        "batch": lambda n: bind.a3d_batch_udf_workspace_bytes(n, 7),
        "sort": lambda n: lib.a3d_sort_pairs_workspace_bytes(n),
        "batch autotune": lambda n: bind.a3d_batch_autotune_workspace_bytes(min(n, 1 << 24), 7),
    }[name]
    ns = sizes()
    got = [size(n) for n in ns]
    falls = [(a, b) for a, b, x, y in zip(ns, ns[1:], got, got[1:]) if y < x]
    assert not falls, falls
