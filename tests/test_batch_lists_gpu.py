"""Batched inserts without per-key flags, where tables of several regions (256 probe groups each) are built from lists
of their regions' keys: every kind of table around one region, several regions, 1024 regions (the most that are built)
and above; out-of-band keys; keys that spill over a region's end, into the next region and around the table's end, and
more of them than the spill buffer takes; a key repeated past a list's length; tables filled past max_size().
What every slot of a table holds, the sizes, the refused inserts and the lookups are those of a dict per table."""

import numpy as np
import pytest
import torch

import oracle as O
import stdgpu_gb300 as sg
from stdgpu_gb300.containers import _DeviceArray

from gpu_util import dev, host

pytestmark = pytest.mark.gpu

REGION, REGIONS, SPILLS = 256, 1024, 1 << 15  # kRegionGroups, kListRegions, kSpillMax
KINDS = [O.SET_U32, O.SET_U64, O.MAP_U64_U32, O.MAP_U64_U64, O.MAP_U32_U32, O.MAP_U32_U64]
SLOT = {O.SET_U32: 4, O.SET_U64: 8, O.MAP_U64_U32: 16, O.MAP_U64_U64: 16, O.MAP_U32_U32: 8, O.MAP_U32_U64: 16}
NAME = {np.dtype(np.uint32): "u32", np.dtype(np.uint64): "u64"}


def _names(kind):
    vd = O.VAL_DTYPE[kind]
    return NAME[np.dtype(O.KEY_DTYPE[kind])], (None if vd is None else NAME[np.dtype(vd)])


def _geometry(kind, cap):
    return sg.geometry_for(sg.KINDS[_names(kind)], int(cap))


def _cap_with_groups(kind, groups):
    """The smallest capacity whose table has at least `groups` probe groups."""
    lo, hi = 1, groups * 128 // SLOT[kind]
    while lo < hi:
        mid = (lo + hi) // 2
        if _geometry(kind, mid).num_groups >= groups:
            hi = mid
        else:
            lo = mid + 1
    return lo


def _home(kind, cap, keys):
    """Home probe group of each key."""
    g = _geometry(kind, cap)
    bits = int(g.bucket_count).bit_length() - 1
    k = keys.astype(np.uint64)
    if bits == 0:
        return np.zeros(len(k), np.int64)
    drop = np.uint64(64 - bits)
    with np.errstate(over="ignore"):
        bucket = ((k ^ (k >> drop)) * np.uint64(11400714819323198485)) >> drop
    return ((bucket * np.uint64(g.num_groups)) >> np.uint64(bits)).astype(np.int64)


def _random(kind, n, rng):
    kd = np.dtype(O.KEY_DTYPE[kind])
    return np.unique(rng.integers(1, np.iinfo(kd).max - 1, size=n + n // 8 + 8, dtype=np.uint64).astype(kd))[:n]


def _near(kind, cap, first, last, count, rng):
    """`count` distinct keys whose home group lies in [first, last)."""
    out = np.zeros(0, O.KEY_DTYPE[kind])
    while len(out) < count:
        k = _random(kind, 1 << 20, rng)
        h = _home(kind, cap, k)
        out = np.unique(np.concatenate([out, k[(h >= first) & (h < last)]]))
    return rng.permutation(out)[:count]


def _stored(b, kind, t):
    """{key: mapped value} of table t's slot image; a key stored twice fails."""
    v = b.view(t)
    raw = torch.as_tensor(_DeviceArray(v.slots, (int(v.num_groups) + 1) * 16, 8), device="cuda").cpu().numpy()
    sb = SLOT[kind]
    rows = raw.view(np.uint8).reshape(-1, sb)
    kd, vd = np.dtype(O.KEY_DTYPE[kind]), O.VAL_DTYPE[kind]
    top = np.iinfo(kd).max
    keys = np.ascontiguousarray(rows[:, : kd.itemsize]).view(kd).ravel()
    n = int(v.num_groups) * (128 // sb)
    live = np.nonzero(keys[:n] < top - kd.type(1))[0]
    vals = keys[live]
    if vd is not None:
        at = 4 if sb == 8 else 8
        vals = np.ascontiguousarray(rows[:, at: at + np.dtype(vd).itemsize]).view(vd).ravel()[live]
    assert len(np.unique(keys[live])) == len(live), t
    assert (keys[int(v.total_count):n] == top - kd.type(1)).all(), t  # the erased marker at and above total_count
    return dict(zip(keys[live].tolist(), vals.tolist()))


def _refused(b, t):
    return int(torch.as_tensor(_DeviceArray(b.view(t).header, 8, 8), device="cuda")[1].item())


def _value(kind, keys):
    vd = O.VAL_DTYPE[kind]
    return None if vd is None else (keys >> keys.dtype.type(1)).astype(vd)


def _insert_and_check(kind, caps, keys, full=()):
    """One insert into fresh tables without flags; tables in `full` get more distinct keys than they take."""
    ks, ms = _names(kind)
    kd, vd = np.dtype(O.KEY_DTYPE[kind]), O.VAL_DTYPE[kind]
    top = np.iinfo(kd).max
    b = sg.table_batch.createDeviceObjects(caps, key=ks, mapped=ms)
    flat = np.concatenate(keys).astype(kd)
    off = np.concatenate([[0], np.cumsum([len(k) for k in keys])]).astype(np.int64)
    vals = _value(kind, flat)
    for _ in range(2):  # again after a clear
        b.insert(dev(flat), dev(off), dev(vals) if vals is not None else None)
        sizes = b.sizes()
        got, found = b.find(dev(flat), dev(off))
        found = found.cpu().numpy()
        for t, cap in enumerate(caps):
            k = keys[t]
            lo, hi = off[t], off[t + 1]
            want = {int(x): int(y) for x, y in zip(k, k if vd is None else _value(kind, k)) if x < top - kd.type(1)}
            special = len(set(k.tolist()) & {int(top), int(top) - 1})
            held = _stored(b, kind, t)
            if t in full:
                room = _geometry(kind, cap).max_size
                assert len(held) == room and sizes[t] == room + special, t
                assert all(want[x] == y for x, y in held.items()), t
                assert _refused(b, t) == len(want) - room, t
                assert np.array_equal(found[lo:hi].astype(bool), [x in held or x >= top - 1 for x in k.tolist()]), t
            else:
                assert held == want and sizes[t] == len(want) + special, t
                assert found[lo:hi].all() and _refused(b, t) == 0, t
                if vd is not None:
                    assert np.array_equal(host(got, vd)[lo:hi], _value(kind, k)), t
        b.clear()
        assert b.sizes().sum() == 0
    sg.table_batch.destroyDeviceObjects(b)


@pytest.mark.parametrize("kind", KINDS)
def test_tables_around_one_region_and_several(kind):
    rng = np.random.default_rng(kind)
    above = _cap_with_groups(kind, REGION + 1)  # (a table of exactly 256 groups does not exist)
    caps = [1, 40, above - 1, above] + [_cap_with_groups(kind, g) for g in (3 * REGION, 5 * REGION - 3, 9 * REGION + 1)]
    assert _geometry(kind, above - 1).num_groups <= REGION
    keys = []
    for c in caps:
        k = _random(kind, max(1, c // 2), rng)
        top = np.iinfo(k.dtype).max
        k = np.concatenate([k, k[: len(k) // 4], np.array([top, top - 1, top], k.dtype)])  # copies, out-of-band keys
        keys.append(rng.permutation(k))
    _insert_and_check(kind, caps, keys)


@pytest.mark.parametrize("kind", [O.SET_U64, O.MAP_U64_U64])
@pytest.mark.parametrize("built", [True, False])
def test_tables_of_the_most_regions_that_are_built(kind, built):
    cap = _cap_with_groups(kind, REGIONS * REGION + 1) - int(built)
    assert (_geometry(kind, cap).num_groups <= REGIONS * REGION) == built
    rng = np.random.default_rng(50)
    _insert_and_check(kind, [cap, 5000], [_random(kind, cap // 3, rng), _random(kind, 3000, rng)])


@pytest.mark.parametrize("kind", KINDS)
def test_keys_that_spill_out_of_built_regions(kind):
    rng = np.random.default_rng(10 + kind)
    cap = _cap_with_groups(kind, 3 * REGION + 7)
    groups = _geometry(kind, cap).num_groups
    slots = 8 * 128 // SLOT[kind]  # of eight groups
    crowd = _near(kind, cap, REGION - 8, REGION, 3 * slots, rng)       # on into region 1
    end = _near(kind, cap, groups - 5, groups, 3 * slots, rng)         # around the table's end, into group 0
    rest = _random(kind, cap // 4, rng)
    keys = [rng.permutation(np.concatenate([rest, crowd, end, crowd])), rest[:1000].copy()]
    _insert_and_check(kind, [cap, _cap_with_groups(kind, REGION)], keys)


def test_more_spilled_keys_than_the_buffer_takes():
    kind = O.SET_U64
    rng = np.random.default_rng(20)
    cap = _cap_with_groups(kind, 3 * REGION)
    crowd = _near(kind, cap, REGION - 8, REGION, REGION * 16, rng)  # a list's length; 128 of them fit the region
    tables = SPILLS // (len(crowd) - 8 * 16) + 3
    _insert_and_check(kind, [cap] * tables, [rng.permutation(crowd) for _ in range(tables)])


@pytest.mark.parametrize("kind", [O.SET_U32, O.SET_U64, O.MAP_U64_U32, O.MAP_U32_U32])
def test_a_key_repeated_past_a_lists_length(kind):
    rng = np.random.default_rng(30)
    cap = _cap_with_groups(kind, 3 * REGION)
    k = _random(kind, cap // 3, rng)
    length = REGION * 128 // SLOT[kind]
    _insert_and_check(kind, [cap, cap], [rng.permutation(np.concatenate([k, np.full(2 * length, k[0])])), k])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("groups", [3, REGION, 2 * REGION + 9])
def test_tables_filled_past_max_size_count_each_refused_key_once(kind, groups):
    rng = np.random.default_rng(40 + groups)
    cap = _cap_with_groups(kind, groups)
    room = _geometry(kind, cap).max_size
    more = _random(kind, room + 20, rng)
    _insert_and_check(kind, [cap, cap], [rng.permutation(more), rng.permutation(more[: room // 2])], full=(0,))


def _microseconds(call, before):
    best = float("inf")
    for _ in range(5):
        before()
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        call()
        end.record()
        end.synchronize()
        best = min(best, start.elapsed_time(end) * 1e3)
    return best


@pytest.mark.parametrize("tables", [1, 8])
def test_many_copies_for_few_small_tables_are_not_left_to_one_block_each(tables):
    """The first insert into a cleared table costs about what the same insert costs on a table that holds the keys:
    one block that took all of a table's keys by itself would take far longer than the whole chip."""
    per = (1 << 22) // tables
    keys = torch.arange(1, 501, device="cuda").repeat(1 + per // 500)[:per].repeat(tables)
    off = torch.arange(tables + 1, dtype=torch.int64, device="cuda") * per
    b = sg.table_batch.createDeviceObjects([1000] * tables, key="u64")
    first = _microseconds(lambda: b.insert(keys, off), b.clear)
    assert b.sizes().tolist() == [500] * tables
    again = _microseconds(lambda: b.insert(keys, off), lambda: None)
    sg.table_batch.destroyDeviceObjects(b)
    assert first < 5 * again + 50, (first, again)


def test_a_first_insert_that_builds_nothing_costs_little_more_than_the_next():
    """Three keys into each of very many cleared tables: deciding that none is built is a small part of the call."""
    tables = 1 << 16
    keys = torch.arange(1, 3 * tables + 1, device="cuda")
    off = torch.arange(tables + 1, dtype=torch.int64, device="cuda") * 3
    b = sg.table_batch.createDeviceObjects([2100] * tables, key="u64")
    first = _microseconds(lambda: b.insert(keys, off), b.clear)
    assert (b.sizes() == 3).all()
    again = _microseconds(lambda: b.insert(keys, off), lambda: None)
    sg.table_batch.destroyDeviceObjects(b)
    assert first < 1.9 * again, (first, again)


@pytest.mark.parametrize("cap", [300, 30000])
def test_a_batch_makes_few_device_allocations(cap):
    """Creating a batch takes a handful of allocations, each some tens of microseconds of the host's time."""
    before = sg.live_device_allocations()
    b = sg.table_batch.createDeviceObjects([cap] * 64, key="u64")
    assert sg.live_device_allocations() - before <= 7
    sg.table_batch.destroyDeviceObjects(b)
    assert sg.live_device_allocations() == before


@pytest.mark.parametrize("kind,size", [(k, "regions") for k in KINDS] + [
    (O.SET_U64, "many"), (O.SET_U32, "no regions"), (O.MAP_U64_U32, "no regions")])
def test_clear_leaves_every_slot_and_header_as_new(kind, size):
    """One launch over the regions clears a batch of up to 256 MB; a fill and a launch a larger one (ten tables of the
    most regions) and one with a table that has no regions."""
    most = _cap_with_groups(kind, REGIONS * REGION + 1)
    caps = {"regions": [_cap_with_groups(kind, 5 * REGION + 3), 1, 300, _cap_with_groups(kind, REGION + 1), 77],
            "many": [most - 1] * 10 + [5], "no regions": [100, most, 2000]}[size]
    arena = sum(_geometry(kind, c).num_groups + 1 for c in caps) * 128
    assert (arena > 1 << 28) == (size == "many")
    ks, ms = _names(kind)
    kd, vd = np.dtype(O.KEY_DTYPE[kind]), O.VAL_DTYPE[kind]
    top = np.iinfo(kd).max
    rng = np.random.default_rng(kind)
    keys = [np.concatenate([_random(kind, min(c, 20000), rng), np.array([top, top - 1], kd)]) for c in caps]
    flat = np.concatenate(keys)
    off = np.concatenate([[0], np.cumsum([len(k) for k in keys])]).astype(np.int64)
    vals = _value(kind, flat)
    b = sg.table_batch.createDeviceObjects(caps, key=ks, mapped=ms)
    for _ in range(2):
        b.insert(dev(flat), dev(off), dev(vals) if vals is not None else None)
        b.erase(dev(flat[: len(keys[0]) // 2]), dev(np.minimum(off, len(keys[0]) // 2)))
        b.clear()
        for t in range(len(caps)):
            assert _stored(b, kind, t) == {}, t
            v = b.view(t)
            raw = torch.as_tensor(_DeviceArray(v.slots, (int(v.num_groups) + 1) * 16, 8), device="cuda").cpu().numpy()
            rows = np.ascontiguousarray(raw.view(np.uint8).reshape(-1, SLOT[kind])[:, : kd.itemsize]).view(kd).ravel()
            assert (rows[: int(v.total_count)] == top).all(), t
            assert (rows[int(v.num_groups) * (128 // SLOT[kind]):] == top).all(), t
            assert not torch.as_tensor(_DeviceArray(v.header, 8, 8), device="cuda").any().item(), t
        assert not b.contains(dev(flat), dev(off)).any().item() and b.sizes().sum() == 0
    sg.table_batch.destroyDeviceObjects(b)


def test_clearing_a_small_batch_costs_about_what_clearing_a_table_costs():
    """One launch either way: a fill of the arena and a launch behind it took a small batch several times as long."""
    def each(clear):
        def calls():
            for _ in range(20):
                clear()
        return _microseconds(calls, lambda: torch.cuda._sleep(2_000_000)) / 20  # queued behind a sleeping kernel

    b = sg.table_batch.createDeviceObjects([1000] * 64, key="u64")
    t = sg.unordered_set.createDeviceObject(1000, key="u64")
    batch, table = each(b.clear), each(t.clear)
    sg.table_batch.destroyDeviceObjects(b)
    sg.unordered_set.destroyDeviceObject(t)
    assert batch < 3 * table, (batch, table)
