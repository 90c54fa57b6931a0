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
