"""Calls of several launches of which the runtime refuses one: the call reports it, and what it left behind changes
nothing for the calls after it.  The refusal is made on the host, by a library preloaded before the CUDA runtime
(tests/cpp/refuse_launch.c); no kernel fails."""

import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PRELUDE = r'''
import ctypes, os, sys
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
import torch
import stdgpu_gb300 as sg
from stdgpu_gb300 import _native as N
refuse = ctypes.CDLL(os.environ["LD_PRELOAD"]).refuse_launch
MIX = -7046029254386353131
def keys(lo, n):
    return (torch.arange(lo + 1, lo + n + 1, device="cuda") * MIX) & 0x7FFFFFFFFFFFFFFF
def refused(k, call):
    """The call with its k-th launch refused; whether it said so."""
    refuse(k)
    try:
        call()
    except N.StdgpuError as e:
        refuse(-1)
        assert e.status == N.SG_ERR_CUDA, e.status
        return True
    refuse(-1)
    return False
'''


def _run(scenario):
    lib = ROOT / "tests" / "cpp" / "_build" / "librefuse_launch.so"
    lib.parent.mkdir(exist_ok=True)
    r = subprocess.run(["gcc", "-O1", "-shared", "-fPIC", str(ROOT / "tests" / "cpp" / "refuse_launch.c"), "-o",
                        str(lib), "-ldl"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([sys.executable, "-c", PRELUDE + scenario + '\nprint("OK")', str(ROOT)], capture_output=True,
                       text=True, timeout=300, env=dict(os.environ, LD_PRELOAD=str(lib)))
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr


def test_counted_insert_that_broke_off_leaves_no_candidates_or_bounds():
    """Excess-list accounting, more keys than one launch takes: the keys of the next call get the buckets' own slots
    and the excess slots that they get in a table without the call that broke off."""
    _run(r'''
def excess(t):
    x = ctypes.c_int64()
    N.check(N.load().sg_unordered_excess_used(t._h, None, ctypes.byref(x)), "excess_used")
    return x.value
for at in (0, 1, 2):
    a, b = (sg.unordered_set.createDeviceObject(60000, key="u64") for _ in range(2))
    for t in (a, b):
        t.insert(keys(0, 9000))
    assert refused(at, lambda: a.insert(keys(200000, 20000)))
    done = a.size() - 9000          # launched before the refusal: all of the call's keys, or none
    assert done == (20000 if at == 2 else 0), done
    if at == 2:
        b.insert(keys(200000, 20000))
    more = keys(100000, 25000)
    fa, fb = (torch.zeros(25000, dtype=torch.uint8, device="cuda") for _ in range(2))
    a.insert(more, flags=fa)
    b.insert(more, flags=fb)
    assert bool((fa == 1).all()) and bool((fb == 1).all())
    assert a.size() == b.size() and excess(a) == excess(b), (excess(a), excess(b))
    assert a.valid() and b.valid()
    a.insert(keys(300000, 100))     # a call of one launch
    assert a.size() == b.size() + 100
''')


def test_mixed_deque_call_that_broke_off_leaves_the_deque_as_it_was():
    """A ring too large for turn words, whose mixed calls are a plan and three moves: with any of the four refused the
    counters are as before the call, and the elements are there in order."""
    _run(r'''
cap, n = (1 << 17) + 5, 50000
d = sg.deque.createDeviceObject(cap, elem_bytes=8)
first = torch.arange(1, 30001, device="cuda")
some = torch.arange(n, device="cuda").remainder(3).eq(0).to(torch.uint8)  # more pops than pushes
for kind in (some, 1 - some):
    for at in (0, 1, 2, 3):
        d.clear()
        d.push_back(first)
        assert refused(at, lambda: d.ops(kind, torch.arange(n, device="cuda")))
        assert d.size() == 30000
        vals, ok = d.pop_front(30001)
        assert torch.equal(vals[:30000], first) and int(ok.sum()) == 30000 and d.size() == 0
        d.push_back(first)
        popped, done = d.ops(kind, torch.arange(n, device="cuda") + 10 ** 6)
        pushes, pops = int(kind.sum()), n - int(kind.sum())
        assert d.size() == max(0, 30000 + pushes - pops)
        # more elements than slots, by turn words, which the plan's counts have lain over
        d.clear()
        big = torch.ones(cap + 100, dtype=torch.uint8, device="cuda")
        big[: 60] = 0
        popped, done = d.ops(big, torch.arange(cap + 100, device="cuda"))
        assert d.size() <= cap and d.size() >= cap - 60
''')


def test_batched_insert_that_broke_off_is_not_taken_for_tables():
    """Tables of several regions, whose keys are listed in their own slots before they are built: with the launch that
    builds them refused the batch answers nothing until clear(); with another one refused it goes on."""
    _run(r'''
tables, per = 5, 5000
k = keys(0, tables * per)
off = torch.arange(tables + 1, dtype=torch.int64, device="cuda") * per
b = sg.table_batch.createDeviceObjects([10000] * tables, key="u64")
for at in (0, 1, 2, 3, 4):  # choose, lists, build, tiles, walk
    b.clear()
    assert refused(at, lambda: b.insert(k, off))
    if at == 2:
        for call in (lambda: b.contains(k, off), lambda: b.find(k, off), lambda: b.insert(k, off),
                     lambda: b.erase(k, off)):
            try:
                call()
                raise SystemExit("answered")
            except N.StdgpuError as e:
                assert e.status == N.SG_ERR_CUDA
        b.clear()
    b.insert(k, off)
    assert b.sizes().tolist() == [per] * tables and bool(b.contains(k, off).all())
    assert not bool(b.contains(k + 1, off).any())
''')
