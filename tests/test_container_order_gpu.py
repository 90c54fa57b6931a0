"""The order of bulk calls on one vector or deque, whatever streams they are queued on: calls act in the order in which
the host made them, so a list that takes the same calls one after another holds what the container holds.  Streams are
held back by a sleeping kernel so that a call queued later would otherwise run first."""

from collections import deque as pydeque

import pytest
import torch

import stdgpu_gb300 as sg

pytestmark = pytest.mark.gpu


def _held_back(stream, on):
    if on:
        with torch.cuda.stream(stream):
            torch.cuda._sleep(2_000_000)  # about a millisecond


@pytest.mark.parametrize("n", [1, 700, 5000, 1 << 21])
def test_vector_calls_on_two_streams_act_in_call_order(n):
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    v = sg.vector.createDeviceObject(5 * n, elem_bytes=8)
    parts = [torch.arange(k * n, (k + 1) * n, device="cuda") for k in range(6)]
    torch.cuda.synchronize()
    _held_back(a, True)
    v.push_back(parts[0], stream=a)
    v.push_back(parts[1], stream=b)
    v.push_back(parts[2], stream=a)
    vals, ok = v.pop_back(n, stream=b)
    v.push_back(parts[3], stream=a)
    v.push_back(parts[4], stream=b)
    v.push_back(parts[5], stream=a)
    last = torch.empty(n, dtype=torch.uint8, device="cuda")
    v.push_back(parts[5], flags=last, stream=b)  # full: all fail
    torch.cuda.synchronize()
    assert bool(ok.all()) and torch.equal(vals.sort().values, parts[2])
    assert v.size() == 5 * n and not bool(last.any())
    held, ok = v.pop_back(5 * n)
    assert torch.equal(held.sort().values, torch.cat(parts[:2] + parts[3:]))
    v.clear(stream=a)
    v.push_back(parts[0], stream=b)
    torch.cuda.synchronize()
    assert v.size() == n
    sg.vector.destroyDeviceObject(v)


@pytest.mark.parametrize("cap,n", [(64, 9), (1 << 16, 3000), ((1 << 17) + 3, 20000), (1 << 22, 1 << 20)])
@pytest.mark.parametrize("hold", [0, 1])
def test_deque_calls_on_two_streams_act_in_call_order(cap, n, hold):
    """A producer's and a consumer's stream, both ends, mixed calls whose order is settled, and clear()."""
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    d = sg.deque.createDeviceObject(cap, elem_bytes=8)
    model = pydeque()
    ids = torch.arange(3 * n, device="cuda")
    mixed = torch.arange(n, device="cuda").remainder(3).eq(0).to(torch.uint8)
    torch.cuda.synchronize()
    results = []

    def run(k, call):
        _held_back(streams[k], k == hold)
        results.append(call(streams[k]))

    run(0, lambda s: d.push_back(ids[:n], stream=s))
    run(1, lambda s: d.pop_front(n // 2, stream=s))
    run(0, lambda s: d.push_back(ids[n:2 * n], stream=s))
    run(1, lambda s: d.push_front(ids[2 * n:], stream=s))
    run(0, lambda s: d.pop_back(n // 3, stream=s))
    run(1, lambda s: d.ops(mixed, ids[:n], stream=s))
    run(0, lambda s: d.pop_front(n // 2, stream=s))
    torch.cuda.synchronize()
    host = [int(x) for x in ids.tolist()]
    model.extend(host[:n])
    front = [model.popleft() for _ in range(n // 2)]
    assert results[1][0].tolist() == front and bool(results[1][1].all())
    model.extend(host[n:2 * n])
    for x in host[2 * n:]:
        model.appendleft(x)
    back = [model.pop() for _ in range(n // 3)]
    assert results[4][0].tolist() == back and bool(results[4][1].all())
    # the mixed call has more elements in store than it pops, and room for what it pushes
    pushes = [i for i in range(n) if mixed[i].item()] if n < 4000 else mixed.nonzero().flatten().tolist()
    popped = [model.popleft() for _ in range(n - len(pushes))]
    vals, ok = results[5]
    assert bool(ok.all()) and sorted(vals[mixed == 0].tolist()) == sorted(popped)
    model.extend(host[i] for i in pushes)
    front = [model.popleft() for _ in range(n // 2)]
    assert results[6][0].tolist() == front
    assert d.size() == len(model)
    rest, ok = d.pop_front(len(model) + 1, stream=streams[1])
    torch.cuda.synchronize()
    assert sorted(rest[:-1].tolist()) == sorted(model) and int(ok.sum()) == len(model)
    run(0, lambda s: d.clear(stream=s))
    run(1, lambda s: d.push_back(ids[:n], stream=s))
    torch.cuda.synchronize()
    assert d.size() == n
    sg.deque.destroyDeviceObject(d)


@pytest.mark.parametrize("cap", [5000, 1 << 18])
def test_container_calls_captured_and_made_eagerly_in_turn(cap):
    """A graph of vector and deque calls replayed between calls made on the stream."""
    n = cap // 4
    v = sg.vector.createDeviceObject(cap, elem_bytes=8)
    d = sg.deque.createDeviceObject(cap, elem_bytes=8)
    ids = torch.arange(1, n + 1, device="cuda")
    buf = torch.zeros_like(ids)
    mixed = torch.arange(n, device="cuda").remainder(2).to(torch.uint8)
    out = torch.zeros((3, n), dtype=torch.int64, device="cuda")

    def chain(s):
        v.clear(stream=s)
        d.clear(stream=s)
        buf.copy_(ids)
        v.push_back(buf, stream=s)
        d.push_back(buf, stream=s)
        buf.zero_()
        out[0].copy_(v.pop_back(n, stream=s)[0])
        buf.copy_(ids + n)
        popped, _ = d.ops(mixed, buf, stream=s)
        buf.zero_()
        out[1].copy_(popped)
        out[2].copy_(d.pop_front(n, stream=s)[0])

    def check():
        torch.cuda.synchronize()
        pops = n - int(mixed.sum())
        assert torch.equal(out[0].sort().values, ids)
        assert torch.equal(out[1][mixed == 0].sort().values, ids[:pops])
        want = torch.cat([ids[pops:], (ids + n)[mixed == 1]])
        assert torch.equal(out[2].sort().values, want.sort().values)
        assert v.size() == 0 and d.size() == 0

    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        chain(s)
    check()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        chain(torch.cuda.current_stream())
    for _ in range(3):
        out.zero_()
        g.replay()
        check()
        v.push_back(ids)
        d.push_back(ids)
        torch.cuda.synchronize()
        assert v.size() == n and d.size() == n
    sg.vector.destroyDeviceObject(v)
    sg.deque.destroyDeviceObject(d)


@pytest.mark.parametrize("n", [300, 5000, 1 << 20])
def test_early_kernels_behind_another_streams_work(n):
    """Inputs written on another stream directly before an event that the call's stream waits for, with other early
    calls queued on that stream before: the calls see the inputs."""
    other, s = torch.cuda.Stream(), torch.cuda.Stream()
    t = sg.unordered_set.createDeviceObject(2 * n, key="u64")
    v = sg.vector.createDeviceObject(4 * n, elem_bytes=8)
    d = sg.deque.createDeviceObject(4 * n, elem_bytes=8)
    b = sg.table_batch.createDeviceObjects([4 * n] * 3, key="u64")
    src = torch.arange(1, n + 1, device="cuda") * 0x9E3779B97F4A7C1
    buf = torch.zeros_like(src)
    off = torch.tensor([0, 0, n, n], device="cuda")
    torch.cuda.synchronize()
    for _ in range(3):
        with torch.cuda.stream(other):
            torch.cuda._sleep(1_000_000)
            buf.copy_(src)
        done = torch.cuda.Event()
        done.record(other)
        with torch.cuda.stream(s):
            t.clear(stream=s)
            v.clear(stream=s)
            d.clear(stream=s)
            b.clear(stream=s)
            s.wait_event(done)
            t.insert(buf, stream=s)
            v.push_back(buf, stream=s)
            d.push_back(buf, stream=s)
            b.insert(buf, off, stream=s)
            got = t.contains(src, stream=s), b.contains(src, off, stream=s), d.pop_front(n, stream=s)[0]
            buf.zero_()
        s.synchronize()
        assert bool(got[0].all()) and bool(got[1].all()) and torch.equal(got[2], src)
        assert t.size() == n and v.size() == n and b.sizes().tolist() == [0, n, 0]
    sg.unordered_set.destroyDeviceObject(t)
    sg.vector.destroyDeviceObject(v)
    sg.deque.destroyDeviceObject(d)
    sg.table_batch.destroyDeviceObjects(b)


@pytest.mark.parametrize("cap", [4096, 1 << 18])
def test_clear_makes_a_container_whole_whatever_its_launch_words_hold(cap):
    """A graph replayed while a call runs on the same object can leave the count of arrived blocks behind, and then no
    later call ends properly: clear() starts it anew.  Here the words are written from the host."""
    import ctypes
    from stdgpu_gb300 import _native as N
    from stdgpu_gb300.containers import _DeviceArray
    n = cap // 4
    ids = torch.arange(1, n + 1, device="cuda")
    v = sg.vector.createDeviceObject(n, elem_bytes=8)
    d = sg.deque.createDeviceObject(cap, elem_bytes=8)
    view, dview = N.sg_vector_view(), N.sg_deque_view()
    N.check(N.load().sg_vector_view_of(v._h, ctypes.byref(view)), "view")
    N.check(N.load().sg_deque_view_of(d._h, ctypes.byref(dview)), "view")
    for sync in (view.sync, dview.sync):  # the words of the launches lie behind the device calls' own, at 64
        torch.as_tensor(_DeviceArray(sync + 64, 16, 4), device="cuda").fill_(3)
    torch.cuda.synchronize()
    v.clear()
    d.clear()
    v.push_back(torch.cat([ids, ids]))
    raw = torch.as_tensor(_DeviceArray(view.size, 1, 8), device="cuda")
    assert int(raw[0].item()) == n  # clamped by the call's last block
    vals, ok = v.pop_back(n)
    assert bool(ok.all()) and v.size() == 0
    d.push_back(ids)
    d.ops(torch.ones(n, dtype=torch.uint8, device="cuda"), ids)
    assert d.size() == 2 * n and torch.equal(d.pop_front(n)[0], ids)
    sg.vector.destroyDeviceObject(v)
    sg.deque.destroyDeviceObject(d)


@pytest.mark.parametrize("before", ["nothing", "kernel", "copy", "memset", "fork"])
@pytest.mark.parametrize("n", [300, 5000, 1 << 20])
def test_early_kernels_captured_behind(before, n):
    """The first call of a captured graph behind each kind of work: nothing, a kernel, a copy, a memset, and a kernel
    together with another stream's that was joined by an event."""
    t = sg.unordered_map.createDeviceObject(2 * n, key="u64", mapped="u32")
    v = sg.vector.createDeviceObject(n, elem_bytes=8)
    d = sg.deque.createDeviceObject(4 * n, elem_bytes=8)
    b = sg.table_batch.createDeviceObjects([4 * n] * 2, key="u64")
    src = torch.arange(1, n + 1, device="cuda") * 0x9E3779B97F4A7C1
    vals = torch.arange(n, dtype=torch.int32, device="cuda")
    off = torch.tensor([0, n, n], device="cuda")
    keys, other, spare = torch.empty_like(src), torch.empty_like(vals), torch.empty_like(src)
    out = torch.empty((5, n), dtype=torch.int64, device="cuda")
    side = torch.cuda.Stream()

    def work(s):
        """Writes keys and mapped values; the stream's last piece of work is of the kind asked for."""
        if before == "nothing":
            return
        if before == "fork":
            side.wait_stream(s)
            with torch.cuda.stream(side):
                keys.copy_(src)
            torch.mul(vals, 1, out=other)
            s.wait_stream(side)
            return
        torch.mul(src, 1, out=keys)
        torch.mul(vals, 1, out=other)
        if before == "copy":
            keys.copy_(src)
        if before == "memset":
            spare.zero_()

    def calls(s):
        steps = [lambda: t.clear(stream=s), lambda: t.insert(keys, other, stream=s),
                 lambda: out[0].copy_(t.find(keys, stream=s)[0]), lambda: t.erase(keys[: n // 2], stream=s),
                 lambda: out[1].copy_(t.contains(keys, stream=s)),
                 lambda: v.clear(stream=s), lambda: v.push_back(keys, stream=s),
                 lambda: out[2].copy_(v.pop_back(n, stream=s)[0]),
                 lambda: d.clear(stream=s), lambda: d.push_back(keys, stream=s),
                 lambda: out[3].copy_(d.pop_front(n, stream=s)[0]),
                 lambda: b.clear(stream=s), lambda: b.insert(keys, off, stream=s),
                 lambda: out[4].copy_(b.contains(keys, off, stream=s))]
        for step in steps:
            work(s)
            step()

    keys.copy_(src)
    other.copy_(vals)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        calls(s)  # warm-up
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        calls(torch.cuda.current_stream())
    for _ in range(3):
        if before != "nothing":
            keys.zero_()
            other.zero_()
        out.fill_(-1)
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out[0], vals.long())
        assert not bool(out[1][: n // 2].any()) and bool((out[1][n // 2:] == 1).all())
        assert torch.equal(out[2].sort().values, src.sort().values)
        assert torch.equal(out[3], src) and bool((out[4] == 1).all())
        assert t.size() == n - n // 2 and b.sizes().tolist() == [n, 0]
    sg.unordered_map.destroyDeviceObject(t)
    sg.vector.destroyDeviceObject(v)
    sg.deque.destroyDeviceObject(d)
    sg.table_batch.destroyDeviceObjects(b)
