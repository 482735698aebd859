"""The radix sort around its changes of form: two, four, eight and sixteen
keys a thread, the fused digit offsets up to 128 tiles and the scanned ones
above, partial last tiles, 32-bit keys through the query sort's own range, and
keys of few distinct digits (whole warps of one digit).  Exact against a stable
torch sort."""

import pytest
import torch

from atom3d_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["random", "two values", "sorted", "top bits"])
@pytest.mark.parametrize("n", [1, 2, 31, 511, 512, 513, 65536, 65537, 131072, 131073, 606207, 606208, 1212415,
                               1212417])
def test_radix_sort_is_stable(n, kind):
    g = torch.Generator(device="cuda").manual_seed(n)
    keys = torch.randint(0, 2 ** 40, (n,), generator=g, device="cuda", dtype=torch.int64)
    if kind == "two values":
        keys = (keys & 1) * 0xFF00FF00FF
    elif kind == "sorted":
        keys = keys.sort().values >> 20
    elif kind == "top bits":
        keys = keys << 23
    vals = torch.arange(n, device="cuda", dtype=torch.int32)
    ref, order = torch.sort(keys, stable=True)
    ws = _lib.workspace(_lib.lib().a3d_sort_pairs_workspace_bytes(n), keys.device)
    _lib.call("a3d_sort_pairs_u64", keys.data_ptr(), vals.data_ptr(), n, 0, 64, ws.data_ptr(), ws.numel(),
              _lib.stream_ptr(keys.device))
    assert torch.equal(keys, ref)
    assert torch.equal(vals.long(), order)
