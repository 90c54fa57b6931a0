"""range_copy() and device_range() report a wait that gave up in their own call, not in an earlier one: with the error
bit of such a call left in the table's header (written here from the host) they give the whole range, and so does
rehash(), which goes through them."""

import numpy as np
import pytest
import torch

import oracle as O
from stdgpu_gb300.containers import _DeviceArray

from test_unordered_gpu import Table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3000, 2000000])
def test_an_earlier_calls_report_does_not_stay(n):
    t = Table(O.MAP_U64_U32, 2 * n)
    keys = np.arange(1, n + 1, dtype=np.uint64) * np.uint64(2654435761)
    t.insert(keys, (keys >> np.uint64(3)).astype(np.uint32))
    words = torch.as_tensor(_DeviceArray(t.t.view().header, 10, 4), device="cuda")
    for _ in range(2):
        words[8] |= 16  # table_header::error, kErrRange
        got, mapped = t.range()
        assert np.array_equal(np.sort(got), keys)
        assert np.array_equal(mapped, (got >> np.uint64(3)).astype(np.uint32))
        assert int(words[8].item()) == 0
        words[8] |= 16
        assert t.t.device_range().numel() == n
        words[8] |= 16
        t.t.rehash(3 * n)
        words = torch.as_tensor(_DeviceArray(t.t.view().header, 10, 4), device="cuda")
        assert t.size() == n and np.array_equal(np.sort(t.range()[0]), keys)
    t.close()
