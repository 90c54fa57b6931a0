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
