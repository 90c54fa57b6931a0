"""Kernels that are set up while the stream's work before them ends still see all of that work: each call's input is
written on the stream directly before the call and overwritten directly after it, once on the stream and then as a
replayed graph.  The expected flags are whole numbers that follow from the calls, so the check is equality."""

import pytest
import torch

import stdgpu_gb300 as sg

pytestmark = pytest.mark.gpu


def chain(t, src, keys, out):
    """clear, insert the keys, look up twice as many, erase half of them, look the keys up again."""
    n = src.numel() // 2
    st = torch.cuda.current_stream()
    t.clear(stream=st)
    keys[:n].copy_(src[:n])
    t.insert(keys[:n], stream=st)
    keys.zero_()
    keys.copy_(src.flip(0))
    out[0].copy_(t.contains(keys, stream=st))
    keys.zero_()
    keys[: n // 2].copy_(src[: n // 2])
    t.erase(keys[: n // 2], stream=st)
    keys.zero_()
    keys.copy_(src)
    out[1].copy_(t.contains(keys, stream=st))
    keys.zero_()


@pytest.mark.parametrize("n", [2, 700, 4096, 4098, 200000, 3000000])
def test_calls_see_the_stream_before_them(n):
    t = sg.unordered_set.createDeviceObject(n, key="u64")
    src = torch.arange(1, 2 * n + 1, dtype=torch.int64, device="cuda") * 0x9E3779B97F4A7C1
    keys = torch.zeros_like(src)
    out = torch.zeros((2, 2 * n), dtype=torch.uint8, device="cuda")
    want = torch.zeros_like(out)
    want[0, n:] = 1  # the first half of the keys, looked up in reverse order
    want[1, n // 2 : n] = 1
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        for _ in range(2):
            out.fill_(7)
            chain(t, src, keys, out)
            assert torch.equal(out, want) and t.size(stream=s) == n - n // 2
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        chain(t, src, keys, out)
    for _ in range(3):
        out.fill_(7)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want) and t.size() == n - n // 2
    assert t.valid()
    sg.unordered_set.destroyDeviceObject(t)


@pytest.mark.parametrize("n", [1, 513, 70000, (1 << 21) + 5])
def test_container_calls_see_the_stream_before_them(n):
    v = sg.vector.createDeviceObject(2 * n, elem_bytes=8)
    d = sg.deque.createDeviceObject(2 * n, elem_bytes=8)
    src = torch.arange(1, n + 1, dtype=torch.int64, device="cuda")
    mixed = torch.arange(n, device="cuda").remainder(2).to(torch.uint8)
    buf = torch.zeros_like(src)
    pred = torch.zeros(n, dtype=torch.uint8, device="cuda")
    pushes = int(mixed.sum())
    for _ in range(3):
        v.clear()
        d.clear()
        buf.copy_(src)
        pred.copy_(mixed)
        v.push_back(buf, pred)
        pred.zero_()
        d.push_back(buf)
        buf.zero_()
        vals, ok = v.pop_back(pushes)
        assert v.size() == 0 and bool(ok.all()) and torch.equal(vals.sort().values, src[mixed.bool()])
        buf.copy_(src)
        pred.copy_(mixed)
        popped, done = d.ops(pred, buf)  # the pops take the first elements, the pushes go behind them
        buf.zero_()
        pred.zero_()
        assert bool(done.all()) and torch.equal(popped[~mixed.bool()].sort().values, src[: n - pushes])
        vals, ok = d.pop_front(n + 1)
        left = n - (n - pushes) + pushes
        assert int(ok.sum()) == min(left, n + 1) and d.size() == left - int(ok.sum())
        assert torch.equal(vals[: n - (n - pushes)], src[n - pushes :])
    sg.vector.destroyDeviceObject(v)
    sg.deque.destroyDeviceObject(d)


def test_batched_calls_see_the_stream_before_them():
    per, tables = 300, 200
    b = sg.table_batch.createDeviceObjects([per] * tables, key="u64")
    src = torch.arange(1, per * tables + 1, dtype=torch.int64, device="cuda")
    offsets = torch.arange(tables + 1, dtype=torch.int64, device="cuda") * per
    buf, off = torch.zeros_like(src), torch.zeros_like(offsets)
    for _ in range(3):
        b.clear()
        buf.copy_(src)
        off.copy_(offsets)
        b.insert(buf, off)
        buf.copy_(src + per)  # the next table's keys
        none = b.contains(buf, off)
        buf.copy_(src)
        every = b.contains(buf, off)
        off.zero_()
        buf.zero_()
        assert int(none.sum()) == 0 and int(every.sum()) == per * tables
    sg.table_batch.destroyDeviceObjects(b)


@pytest.mark.parametrize("n", [32, 4097, 300000])
def test_lookups_of_hot_keys_see_the_last_calls(n):
    """Queries that repeat few keys, which a lookup may read from the SM's own cache, between calls that store and
    erase those keys."""
    t = sg.unordered_map.createDeviceObject(3000, key="u64", mapped="u32")
    hot = torch.arange(1, 101, dtype=torch.int64, device="cuda") * 0x9E3779B97F4A7C1
    pick = torch.arange(n, device="cuda").remainder(100)
    for call in range(1, 4):
        stored = hot[: 30 * call]
        t.insert(stored, torch.full((30 * call,), call, dtype=torch.int32, device="cuda"))
        vals, found = t.find(hot[pick])
        assert torch.equal(found.bool(), pick < 30 * call)
        assert torch.equal(vals != 0, pick < 30 * call)
        t.erase(stored[:10])
        assert torch.equal(t.contains(hot[pick]).bool(), (pick >= 10) & (pick < 30 * call))
        t.insert(stored[:10], torch.full((10,), 9, dtype=torch.int32, device="cuda"))
        vals, _ = t.find(hot[pick])
        assert torch.equal(vals[pick < 10], torch.full_like(vals[pick < 10], 9))
    sg.unordered_map.destroyDeviceObject(t)
