"""Batched inserts with flags per key into tables that hold nothing.  Tables of one region (256 probe groups) are then
built in shared memory, larger ones take their keys through the probe kernel (without flags they are built from
lists of their regions' keys: tests/test_batch_lists_gpu.py).  Tables of less than a region's groups, about
one region's and several; too few keys to be built; keys crowded into a few neighbouring groups and around the table's
end; tables filled to max_size() and past it; a batch with only some tables empty.  Sizes, flags per key, contents and
lookups equal a dict's per table."""

import numpy as np
import pytest
import torch

import oracle as O
import stdgpu_gb300 as sg

from gpu_util import dev, host, per_key_success

pytestmark = pytest.mark.gpu

MIX = 11400714819323198485


def _names(kind):
    kd, vd = O.KEY_DTYPE[kind], O.VAL_DTYPE[kind]
    return ("u32" if kd == np.uint32 else "u64"), (None if vd is None else "u32" if vd == np.uint32 else "u64")


def _check(b, kind, tables, keys, calls):
    """Inserts each call's keys and compares every table with a Python dict."""
    kd, vd = O.KEY_DTYPE[kind], O.VAL_DTYPE[kind]
    held = [dict() for _ in tables]
    for call in calls:
        per = [keys[t][call[t][0]:call[t][1]] for t in range(len(tables))]
        flat = np.concatenate(per).astype(kd)
        off = np.concatenate([[0], np.cumsum([len(x) for x in per])]).astype(np.int64)
        vals = (flat >> kd(1)).astype(vd) if vd is not None else None
        flags = torch.full((len(flat),), 9, dtype=torch.uint8, device="cuda")
        b.insert(dev(flat), dev(off), dev(vals) if vals is not None else None, flags=flags)
        f = flags.cpu().numpy()
        got, found = b.find(dev(flat), dev(off))
        found = found.cpu().numpy()
        for t in range(len(tables)):
            lo, hi = off[t], off[t + 1]
            new = set(per[t].tolist()) - set(held[t])
            ok = per_key_success(flat[lo:hi], f[lo:hi])
            assert all(ok[k] == (1 if k in new else 0) for k in ok), t
            held[t].update({k: k >> 1 for k in new})
            assert found[lo:hi].all(), t
            if vd is not None:
                assert np.array_equal(host(got, vd)[lo:hi], vals[lo:hi]), t
        assert np.array_equal(b.sizes(), np.array([len(h) for h in held]))
    return held


@pytest.mark.parametrize("kind", [O.SET_U32, O.SET_U64, O.MAP_U64_U32, O.MAP_U32_U32, O.MAP_U32_U64])
def test_built_tables_equal_a_dict(kind):
    rng = np.random.default_rng(kind)
    kd = O.KEY_DTYPE[kind]
    per_group = {O.SET_U32: 32, O.SET_U64: 16, O.MAP_U32_U32: 16}.get(kind, 8)
    caps = [1, 7, 64 * per_group, 320 * per_group, 512 * per_group, 700 * per_group, 2600 * per_group,
            3000 * per_group, 6000 * per_group, 45000 * per_group]
    keys = []
    for c in caps:
        n = max(1, c // 2)
        k = rng.integers(0, np.iinfo(kd).max - 1, size=n, dtype=np.uint64).astype(kd)
        k[n // 2:n // 2 + n // 8] = k[: n // 8]  # copies
        if n > 8:
            k[3], k[4] = np.iinfo(kd).max, np.iinfo(kd).max - 1  # the out-of-band keys
        keys.append(k)
    ks, ms = _names(kind)
    b = sg.table_batch.createDeviceObjects(caps, key=ks, mapped=ms)
    full = [(0, len(k)) for k in keys]
    few = [(0, 1 + len(k) // 200) for k in keys]     # too few keys for most tables: the probe kernel
    half = [(0, len(k) // 2 if t % 2 else 0) for t, k in enumerate(keys)]  # every other table stays empty
    _check(b, kind, caps, keys, [full])
    b.clear()
    _check(b, kind, caps, keys, [few, full])
    b.clear()
    _check(b, kind, caps, keys, [half, full])
    b.clear()
    assert b.sizes().sum() == 0
    sg.table_batch.destroyDeviceObjects(b)


def _keys_near(bits, groups, total_groups, first, last, count, rng):
    """u64 keys whose home group lies in [first, last)."""
    out = []
    while len(out) < count:
        k = rng.integers(0, 1 << 63, size=1 << 18, dtype=np.uint64)
        with np.errstate(over="ignore"):
            bucket = ((k ^ (k >> np.uint64(64 - bits))) * np.uint64(MIX)) >> np.uint64(64 - bits)
        g = (bucket * np.uint64(total_groups)) >> np.uint64(bits)
        out.extend(k[(g >= first) & (g < last)].tolist())
    return np.array(out[:count], dtype=np.uint64)


def test_keys_that_spill_over_a_regions_end():
    """Three times as many keys as slots in 8 neighbouring groups: most go on into the next groups, through the probe
    kernel (the inserts ask for flags), and a small table of the batch is built as usual."""
    cap = 80000
    g = sg.geometry_for(sg.KINDS[("u64", None)], cap)
    assert g.num_groups > 4096 + 64  # room behind the 4096 groups whose end is crowded
    bits = int(g.bucket_count).bit_length() - 1
    rng = np.random.default_rng(5)
    crowd = _keys_near(bits, None, g.num_groups, 4088, 4096, 3 * 8 * 16, rng)
    end = _keys_near(bits, None, g.num_groups, g.num_groups - 8, g.num_groups, 3 * 8 * 16, rng)  # wraps to group 0
    rest = rng.integers(0, 1 << 63, size=20000, dtype=np.uint64)
    keys = [np.concatenate([rest, crowd, end, crowd]), rest[:1000].copy()]
    caps = [cap, 3000]
    b = sg.table_batch.createDeviceObjects(caps, key="u64")
    _check(b, O.SET_U64, caps, keys, [[(0, len(k)) for k in keys]])
    sg.table_batch.destroyDeviceObjects(b)


@pytest.mark.parametrize("cap", [1, 3, 100, 5000, 40000])
def test_tables_filled_past_their_size(cap):
    """More distinct keys than max_size(): exactly max_size() of them are stored, the others refused."""
    g = sg.geometry_for(sg.KINDS[("u64", None)], cap)
    n = g.max_size + 50
    keys = (np.arange(1, n + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)) >> np.uint64(1)
    b = sg.table_batch.createDeviceObjects([cap, 200], key="u64")
    off = np.array([0, n, n + 10], dtype=np.int64)
    flat = np.concatenate([keys, keys[:10]])
    flags = torch.zeros(len(flat), dtype=torch.uint8, device="cuda")
    b.insert(dev(flat), dev(off), flags=flags)
    f = flags.cpu().numpy()
    assert f[:n].sum() == g.max_size and b.sizes().tolist() == [g.max_size, 10]
    assert np.array_equal(b.contains(dev(flat), dev(off)).cpu().numpy(), f)
    sg.table_batch.destroyDeviceObjects(b)
