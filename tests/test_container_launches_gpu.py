"""vector::push_back and the deque's mixed launches at the sizes where their launches change: rows, warps, blocks and
tiles and their remainders, the first size that reserves per 8192 elements, predicates that are not word-aligned,
rings that wrap inside a launch, and mixed launches whose pushes and pops do and do not depend on one another."""

import numpy as np
import pytest
import torch

import stdgpu_gb300 as sg

from gpu_util import dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 127, 128, 1023, 1025, (1 << 21) - 1, 1 << 21, (1 << 21) + 8191, (1 << 22) + 33])
@pytest.mark.parametrize("elem", [4, 8])
def test_push_back_keeps_what_is_selected(n, elem):
    rng = np.random.default_rng(n + elem)
    dt = np.uint32 if elem == 4 else np.uint64
    values = rng.permutation(n).astype(dt)
    for offset, share, cap in [(0, 0.3, n), (1, 0.9, n), (16, 1.0, n), (3, 0.5, max(1, n // 3)), (0, 0.0, n)]:
        pred = np.concatenate([np.zeros(offset, np.uint8), (rng.random(n) < share) * rng.integers(1, 256, n)])
        pred = pred.astype(np.uint8)
        d_pred = dev(pred)[offset:]  # an offset the byte loads cannot take as words
        v = sg.vector.createDeviceObject(cap, elem_bytes=elem)
        flags = torch.full((n,), 9, dtype=torch.uint8, device="cuda")
        v.push_back(dev(values), d_pred, flags=flags)
        want = pred[offset:] != 0
        f = flags.cpu().numpy()
        assert v.size() == min(int(want.sum()), cap) == int(f.sum())
        assert not (f.astype(bool) & ~want).any()
        assert np.array_equal(np.sort(host(v.data(), dt)), np.sort(values[f == 1]))
        v.clear()
        v.push_back(dev(values[: cap]))
        assert v.size() == min(n, cap) and np.array_equal(np.sort(host(v.data(), dt)), np.sort(values[: cap]))
        sg.vector.destroyDeviceObject(v)


class Ring:
    """The rule for mixed calls of at most `cap` elements on rings of more than 2^16 slots: pushes while there is room
    and pops while there are elements, in turn, each kind in element order."""

    def __init__(self, cap):
        self.cap, self.x = cap, []

    def ops(self, is_push, values):
        push, pop = np.nonzero(is_push)[0], np.nonzero(is_push == 0)[0]
        left = len(self.x) + len(push) - len(pop)
        push_ok = push[: len(push) - max(0, left - self.cap)]
        pop_ok = pop[: len(pop) + min(0, left)]
        every = self.x + values[push_ok].tolist()  # in ticket order
        out, ok = np.zeros_like(values), np.zeros(len(values), np.uint8)
        out[pop_ok] = every[: len(pop_ok)]
        ok[push_ok] = ok[pop_ok] = 1
        self.x = every[len(pop_ok):]
        return out, ok


@pytest.mark.parametrize("elem", [4, 8])
@pytest.mark.parametrize("n", [1, 32, 255, 2047, 2048, 2049, 4100, 30001])
def test_mixed_launches_act_in_element_order(n, elem):
    """Mixed launches beside a full, a half full and an empty ring, of one kind only, and through several laps of the
    ring, between launches of every other kind: element by element the model's answers and contents."""
    rng = np.random.default_rng(n * 3 + elem)
    dt = np.uint32 if elem == 4 else np.uint64
    cap = max(3 * n + 7, (1 << 16) + 1 + n % 5)  # larger rings are settled at the start of a launch
    d, m = sg.deque.createDeviceObject(cap, elem_bytes=elem), Ring(cap)
    first = rng.integers(1, 1 << 30, size=cap - n).astype(dt)
    d.push_back(dev(first))
    m.x = first.tolist()
    for lap in range(7):
        is_push = (rng.random(n) < [0.5, 0.2, 0.8][lap % 3]).astype(np.uint8) * np.uint8(3)
        if lap % 2 and n > 3:
            is_push = is_push[: n - 3]
        if lap == 3:
            is_push[:] = 0
        elif lap == 4:
            n_in = min(n, cap - len(m.x) - min(n // 2, cap - len(m.x)))  # the pushes below pass the ring's end
            d.push_back(dev(first[:n_in]))
            m.x += first[:n_in].tolist()
        elif lap in (5, 6):
            d.clear()
            m.x = []
        vals = rng.integers(1, 1 << 30, size=len(is_push)).astype(dt)
        torch.full((2 * n + 64,), -1, dtype=torch.int64, device="cuda")  # what the allocator hands out next
        got, ok = d.ops(dev(is_push), dev(vals))
        want, wok = m.ops(is_push, vals)
        assert np.array_equal(ok.cpu().numpy(), wok) and np.array_equal(host(got, dt), want), lap
        assert d.size() == len(m.x) and np.array_equal(host(d.to_tensor(), dt), np.array(m.x, dt))
        k = cap // 5 + 1
        back, bok = d.pop_back(k)
        take = min(k, len(m.x))
        assert int(bok.sum()) == take and np.array_equal(host(back, dt)[:take], np.array(m.x[::-1][:take], dt))
        m.x = m.x[: len(m.x) - take]
        fr = rng.integers(1, 1 << 30, size=k).astype(dt)
        fit = min(k, cap - len(m.x))
        assert int(d.push_front(dev(fr)).sum()) == fit
        m.x = fr[:fit][::-1].tolist() + m.x
        front, fok = d.pop_front(k)
        take = min(k, len(m.x))
        assert int(fok.sum()) == take and np.array_equal(host(front, dt)[:take], np.array(m.x[:take], dt))
        assert not host(front, dt)[take:].any()
        m.x = m.x[take:]
    d.clear()
    assert d.size() == 0
    sg.deque.destroyDeviceObject(d)


@pytest.mark.parametrize("cap,n", [(5, 100), (64, 5000), (5000, 20000), (70000, 131072), (100000, 131072)])
def test_launches_that_wait_between_launches_that_do_not(cap, n):
    """Launches of more elements than the ring has slots, which are ordered by turn words, between launches that
    leave those out: every launch keeps the multiset and writes 0 where nothing was popped."""
    gen = torch.Generator(device="cuda").manual_seed(cap)
    d = sg.deque.createDeviceObject(cap, elem_bytes=8)
    for it in range(9):
        k = n if it % 3 else max(1, cap // 4)
        share = [0.5, 0.55, 0.45][it % 3]
        is_push = (torch.rand(k, device="cuda", generator=gen) < share).to(torch.uint8)
        vals = torch.randint(1, 1 << 62, (k,), dtype=torch.int64, device="cuda", generator=gen)
        before = d.to_tensor()
        popped, ok = d.ops(is_push, vals)
        after = d.to_tensor()
        assert d.size() == after.numel()  # and no wait gave up
        ip, okb = is_push.bool(), ok.bool()
        assert not popped[ip | ~okb].any()
        lhs = torch.sort(torch.cat([popped[~ip & okb], after])).values
        rhs = torch.sort(torch.cat([before, vals[ip & okb]])).values
        assert torch.equal(lhs, rhs), it
        if it % 2:
            d.push_back(vals[: cap // 2 + 1])
            d.pop_front(cap // 3 + 1)
    sg.deque.destroyDeviceObject(d)
