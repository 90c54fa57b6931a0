"""device_range() and range_copy() against the slot image itself: the stored keys, mapped values and slot indices in
slot order, then the out-of-band keys, at sizes around the tiles of the compaction (1 or 2 KB of slots), for empty,
sparse and full tables and after erases.  src/stdgpu/impl/unordered_base_detail.cuh:136-208."""

import numpy as np
import pytest
import torch

import oracle as O
from stdgpu_gb300.containers import _DeviceArray

from gpu_util import host
from test_unordered_gpu import Table

pytestmark = pytest.mark.gpu

SLOT = {O.SET_U32: 4, O.SET_U64: 8, O.MAP_U64_U32: 16, O.MAP_U64_U64: 16, O.MAP_U32_U32: 8, O.MAP_U32_U64: 16}


def slot_image(t, kind):
    """(key, mapped) of every slot, the two out-of-band ones included."""
    v = t.t.view()
    groups = int(v.num_groups) + 1
    raw = torch.as_tensor(_DeviceArray(v.slots, groups * 16, 8), device="cuda").cpu().numpy().view(np.uint8)
    sb = SLOT[kind]
    rows = raw.reshape(-1, sb)
    kd, vd = np.dtype(O.KEY_DTYPE[kind]), O.VAL_DTYPE[kind]
    keys = np.ascontiguousarray(rows[:, : kd.itemsize]).view(kd).ravel()
    vals = None
    if vd is not None:
        at = 4 if sb == 8 else 8
        vals = np.ascontiguousarray(rows[:, at: at + np.dtype(vd).itemsize]).view(vd).ravel()
    return keys, vals, int(v.num_groups) * (128 // sb)


@pytest.mark.parametrize("kind", range(6))
@pytest.mark.parametrize("target", [1, 2047, 2048, 2049, 4096, 8191, 8193, 40000, 1200000])
def test_range_equals_the_slot_image(kind, target):
    rng = np.random.default_rng(kind * 100 + target)
    kd, vd = O.KEY_DTYPE[kind], O.VAL_DTYPE[kind]
    cap = max(1, int(target / 1.5))  # max_size() near the target
    t = Table(kind, cap)
    top = np.iinfo(kd).max
    for share in (0.0, 0.02, 0.6):
        n = int(cap * share)
        keys = (rng.permutation(4 * cap + 4)[:n].astype(kd) + kd(1)) * kd(2654435761)
        if share > 0.5:
            keys = np.concatenate([keys, np.array([top, top - kd(1)], kd)])  # kept outside the groups
        if len(keys):
            t.insert(keys, (keys >> kd(2)).astype(vd) if vd is not None else None)
            t.erase(keys[: len(keys) // 4])
        image, vals, first_special = slot_image(t, kind)
        live = np.nonzero(image[:first_special] < top - kd(1))[0].tolist()
        want_keys = image[live].tolist()
        for s, k in ((0, top), (1, top - kd(1))):
            if t.contains(np.array([k], kd))[0]:
                live.append(first_special + s)
                want_keys.append(int(k))
        assert len(live) == t.size()
        assert np.array_equal(t.t.device_range().cpu().numpy(), np.array(live, np.int32))
        got, mapped = t.range()
        assert np.array_equal(got, np.array(want_keys, kd))
        if vd is not None:
            assert np.array_equal(mapped, vals[live])
    t.close()
