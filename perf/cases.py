"""The work that is timed when this repository's kernels are tuned: one pass of each case is what a program that
uses the containers does over and over, through the package's public calls.

Nine families, sizes from the benchmark configurations, the tests, or generic:

* ``step``     -- clear a table, fill it, look keys up, take some out, ask its size (a frame of a voxel map).
* ``calls``    -- the same on a small table, with the per-element flags of each call (latency and launches count).
* ``churn``    -- a resident map that takes skewed batches: look-ups, inserts of what is new, erase of what left.
* ``hashed``   -- a set of packed 3 x int16 block coordinates whose buckets come from the caller's spatial hash.
* ``merge``    -- one map copied out and put into another (submap fusion, checkpoints of a live map).
* ``batch``    -- thousands of uneven small tables built and probed together.
* ``worklist`` -- a vector collects the selected elements of a launch, a bitset's occupancy is counted.
* ``queue``    -- a deque takes a launch of mixed push_back and pop_front.
* ``served``   -- a stream of typed requests on resident tables, through the server.

Every output is made of whole numbers and does not depend on the order in which elements that race are stored:
keys that repeat in a call carry the same value, and where a container's order is free (a vector filled by a
launch, the elements a pop launch hands out) the ids it holds are marked in an array by id, as a program that
collects ids does.  Tables are given back when their state goes.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import stdgpu_gb300 as sg
from stdgpu_gb300 import server as sg_server

KEY_BYTES = {"u32": 4, "u64": 8}
MAPPED_BYTES = {"": 0, "u32": 4, "u64": 8}
DTYPE = {"u32": torch.int32, "u64": torch.int64}
KINDS = [("u32", ""), ("u64", ""), ("u64", "u32"), ("u64", "u64"), ("u32", "u32"), ("u32", "u64")]

SPHERES, SHELL, CUBE = 64, 3, 1 << 19


def listed():
    return [
        # the voxel-block map of a large scene, rebuilt, queried at 70 % hits, a quarter dropped
        {"name": "voxel map 2^27 keys", "family": "step", "key": "u64", "mapped": "u32", "capacity": 1 << 28,
         "n": 1 << 27, "queries": 1 << 27, "hits": 0.7, "erase": 0.25, "keys": "voxel"},
        # the plain benchmark set: 2^20 uniform keys, half hits, half erased; fits L2
        {"name": "set u32 2^20 keys", "family": "step", "key": "u32", "mapped": "", "capacity": 1 << 21,
         "n": 1 << 20, "queries": 1 << 20, "hits": 0.5, "erase": 0.5, "keys": "uniform"},
        # a map of a few million entries (a hash join's build and probe side), sizes that are no power of two
        {"name": "map u64/u64 5.2 M keys", "family": "step", "key": "u64", "mapped": "u64", "capacity": 8000003,
         "n": 5200001, "queries": 3300007, "hits": 0.8, "erase": 0.1, "keys": "uniform"},
        # a few hundred keys with flags: every call is latency
        {"name": "small set, 700 keys", "family": "calls", "key": "u64", "mapped": "", "capacity": 1000, "n": 700,
         "queries": 1001},
        # tens of thousands of keys with flags: below the size from which tables stop keeping the excess list
        {"name": "map u32/u32 45 K keys", "family": "calls", "key": "u32", "mapped": "u32", "capacity": 65536,
         "n": 45001, "queries": 60000},
        # a resident map at 0.6 load under Zipf batches
        {"name": "live map, Zipf batches", "family": "churn", "key": "u64", "mapped": "u32", "capacity": 1 << 26,
         "load": 0.6, "batch": 1 << 22, "exponent": 0.99},
        # block coordinates with the caller's hash
        {"name": "block set, spatial hash", "family": "hashed", "key": "u64", "mapped": "", "capacity": 1 << 22,
         "n": 2500001, "queries": 2500001, "hits": 0.5},
        # a submap of some million entries put into another map
        {"name": "map copied into a map", "family": "merge", "key": "u64", "mapped": "u32", "capacity": 1 << 23,
         "n": 3 << 20, "into": 1 << 24, "queries": 3 << 20},
        # many small tables
        {"name": "4096 small sets", "family": "batch", "key": "u64", "mapped": "", "tables": 4096, "median": 2048,
         "hits": 0.5},
        # a frontier of selected ids out of 2^26 threads, beside the count of 2^32 occupancy bits
        {"name": "worklist 2^26, bits 2^32", "family": "worklist", "n": 1 << 26, "share": 0.3, "bits": 1 << 32},
        # a work queue in steady state
        {"name": "queue, 2^24 mixed ops", "family": "queue", "n": 1 << 24},
        # a request stream on resident tables
        {"name": "served stream", "family": "served", "tables": 48, "requests": 96, "least": 4096, "most": 1 << 20,
         "cap_least": 1 << 16, "cap_most": 1 << 22},
    ]


def _spread(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi], odd more often than not."""
    x = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    x = min(max(x, lo), hi)
    return x | 1 if rng.random() < 0.7 and x < hi else x


def draw(rng):
    family = rng.choice(["step", "step", "step", "calls", "calls", "churn", "hashed", "merge", "batch", "worklist",
                         "queue", "served"])
    key, mapped = rng.choice(KINDS)
    c = {"family": family}
    if family == "step":
        cap = _spread(rng, 1 << 14, 1 << 26)
        n = max(64, int(cap * rng.uniform(0.2, 0.65)))
        c |= {"key": key, "mapped": mapped, "capacity": cap, "n": n, "queries": max(64, int(n * rng.uniform(0.3, 1.3))),
              "hits": round(rng.uniform(0.1, 0.95), 2), "erase": round(rng.uniform(0.05, 0.6), 2),
              "keys": rng.choice(["uniform", "voxel"]) if key == "u64" else "uniform"}
    elif family == "calls":
        cap = _spread(rng, 64, 400000)
        n = max(16, int(cap * rng.uniform(0.2, 0.75)))
        c |= {"key": key, "mapped": mapped, "capacity": cap, "n": n, "queries": max(16, int(n * rng.uniform(0.4, 1.5)))}
    elif family == "churn":
        cap = _spread(rng, 1 << 21, 1 << 26)
        c |= {"key": "u64", "mapped": rng.choice(["u32", "u64", ""]), "capacity": cap,
              "load": round(rng.uniform(0.3, 0.8), 2),
              "batch": _spread(rng, 1 << 12, max(1 << 13, cap >> 4)), "exponent": round(rng.uniform(0.6, 1.2), 2)}
    elif family == "hashed":
        cap = _spread(rng, 1 << 12, 1 << 24)
        n = int(cap * rng.uniform(0.2, 0.65))
        c |= {"key": "u64", "mapped": rng.choice(["", "u32"]), "capacity": cap, "n": n,
              "queries": max(64, int(n * rng.uniform(0.3, 1.3))), "hits": round(rng.uniform(0.1, 0.9), 2)}
    elif family == "merge":
        cap = _spread(rng, 1 << 13, 1 << 25)
        n = int(cap * rng.uniform(0.05, 0.6))
        c |= {"key": key, "mapped": mapped, "capacity": cap, "n": n, "into": max(cap, 2 * n),
              "queries": max(64, int(n * rng.uniform(0.2, 1.0)))}
    elif family == "batch":
        c |= {"key": key, "mapped": mapped, "tables": _spread(rng, 64, 4096), "median": _spread(rng, 128, 2048),
              "hits": round(rng.uniform(0.1, 0.9), 2)}
    elif family == "worklist":
        n = _spread(rng, 1 << 12, 1 << 26)
        c |= {"n": n, "share": round(rng.uniform(0.02, 1.0), 2), "bits": _spread(rng, 1 << 12, 1 << 32)}
    elif family == "queue":
        c |= {"n": _spread(rng, 1 << 10, 1 << 24)}
    else:
        least = _spread(rng, 1 << 10, 1 << 13)
        cap = _spread(rng, 1 << 15, 1 << 17)
        c |= {"tables": _spread(rng, 8, 64), "requests": _spread(rng, 16, 96), "least": least,
              "most": _spread(rng, least * 4, 1 << 20), "cap_least": cap, "cap_most": _spread(rng, cap * 2, 1 << 22)}
    return c


# ---------------------------------------------------------------- inputs


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randint(g, high, n):
    return torch.randint(0, int(high), (int(n),), generator=g, device="cuda", dtype=torch.int64)


def _word(x):
    """A Python whole number as a signed 64-bit word."""
    x = int(x) & ((1 << 64) - 1)
    return x - (1 << 64) if x >> 63 else x


def _mix64(x):
    """Seeded bijective mixing of 64-bit words (the splitmix64 finaliser)."""
    x = (x ^ ((x >> 30) & ((1 << 34) - 1))) * -4658895280553007687
    x = (x ^ ((x >> 27) & ((1 << 37) - 1))) * -7723592293110705685
    return x ^ ((x >> 31) & ((1 << 33) - 1))


def _distinct(n, key, seed):
    """n distinct keys that look uniform: a bijection of consecutive numbers."""
    x = torch.arange(n, device="cuda", dtype=torch.int64)
    if key == "u64":
        return _mix64(x + _word(int(seed) * 0x9E3779B97F4A7C15))
    m = (1 << 32) - 1
    x = (x + (int(seed) * 0x9E3779B1 & m)) & m
    x = ((x ^ (x >> 16)) * 0x85EBCA6B) & m
    x = ((x ^ (x >> 13)) * 0xC2B2AE35) & m
    return (x ^ (x >> 16)).to(torch.int32)


def _pack_voxels(x, y, z):
    """21 bits an axis, each offset by 2^20."""
    o = 1 << 20
    return ((x + o) << 42) | ((y + o) << 21) | (z + o)


def _voxels(n, g):
    """n distinct packed block coordinates near the surfaces of a union of spheres, in scan order."""
    centre = torch.randint(-CUBE, CUBE, (SPHERES, 3), generator=g, device="cuda", dtype=torch.int64).double()
    most = 2000.0 if n > 1 << 20 else 400.0
    radius = 50.0 + (most - 50.0) * torch.rand(SPHERES, generator=g, device="cuda", dtype=torch.float64)
    share = torch.cumsum(radius ** 2, 0) / (radius ** 2).sum()
    got = None
    while got is None or got.numel() < n:
        parts = [] if got is None else [got]
        more = int((n - (0 if got is None else got.numel())) * 1.1) + 4096
        for lo in range(0, more, 1 << 25):
            k = min(1 << 25, more - lo)
            s = torch.searchsorted(share, torch.rand(k, generator=g, device="cuda", dtype=torch.float64)).clamp_(max=SPHERES - 1)
            d = torch.randn(3, k, generator=g, device="cuda")
            d = d / d.norm(dim=0).clamp_min(1e-6)
            r = radius[s].float() + (2 * SHELL) * (torch.rand(k, generator=g, device="cuda") - 0.5)
            xyz = [(centre[s, a] + (r * d[a]).double()).round().long() for a in range(3)]
            parts.append(_pack_voxels(*xyz))
            del s, d, r, xyz
        got = torch.unique(torch.cat(parts))
        del parts
    if got.numel() > n:
        got = got[torch.sort(torch.randperm(got.numel(), generator=g, device="cuda")[:n]).values]
    return got


def _queries(keys, absent, n, hits, g):
    """n queries, the given share of them keys that are stored."""
    hit = torch.rand(n, generator=g, device="cuda") < hits
    q = torch.where(hit, keys[_randint(g, keys.numel(), n)], absent[_randint(g, absent.numel(), n)])
    return q.contiguous()


def _values(keys, mapped):
    """A value that is a hash of its key, so that repeated keys carry the same one."""
    return _mix64(keys.long() ^ 0x5DEECE66D).to(DTYPE[mapped]) if mapped else None


def _zipf(n, universe, s, g):
    """Zipf ranks below `universe`, by inversion of the continuous law."""
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    if abs(s - 1.0) < 1e-9:
        r = torch.exp(u * math.log(universe))
    else:
        a = 1.0 - s
        r = (1.0 + u * (float(universe) ** a - 1.0)) ** (1.0 / a)
    return r.floor_().long().clamp_(0, universe - 1)


def _table(case, capacity=None, custom_hash=False):
    cap = int(case["capacity"] if capacity is None else capacity)
    if case["mapped"]:
        return sg.unordered_map.createDeviceObject(cap, key=case["key"], mapped=case["mapped"], custom_hash=custom_hash)
    return sg.unordered_set.createDeviceObject(cap, key=case["key"], custom_hash=custom_hash)


class State:
    """What a program keeps between passes; its containers are given back with it."""

    def __init__(self, case):
        self.case = case
        self.owned = []

    def own(self, obj, destroy):
        self.owned.append((obj, destroy))
        return obj

    def table(self, *a, **k):
        return self.own(_table(self.case, *a, **k), sg.unordered_base.destroyDeviceObject)

    def __del__(self):
        while self.owned:
            obj, destroy = self.owned.pop()
            destroy(obj)


# ---------------------------------------------------------------- step


def _prepare_step(s, c, seed):
    g = _gen(seed)
    n, nq = c["n"], c["queries"]
    extra = max(1024, n // 4)
    if c["keys"] == "voxel":
        every = _voxels(n + extra, g)
        out = torch.zeros(every.numel(), dtype=torch.bool, device="cuda")
        out[torch.randperm(every.numel(), generator=g, device="cuda")[:extra]] = True
        s.keys, absent = every[~out].contiguous(), every[out].contiguous()
        del every, out
    elif c["key"] == "u32":
        both = _randint(g, (1 << 32) - 1, n + extra).to(torch.int32)  # natural repeats among them
        s.keys, absent = both[:n].clone(), both[n:].clone()
    else:
        both = _distinct(n + extra, "u64", seed)
        s.keys, absent = both[:n].clone(), both[n:].clone()
    s.vals = _values(s.keys, c["mapped"])
    s.queries = _queries(s.keys, absent, nq, c["hits"], g)
    s.gone = s.keys[torch.randperm(n, generator=g, device="cuda")[: max(1, int(n * c["erase"]))]].contiguous()
    s.t = s.table()


def _run_step(s):
    t = s.t
    t.clear()
    t.insert(s.keys, s.vals)
    got = t.find(s.queries) if s.case["mapped"] else t.contains(s.queries)
    t.erase(s.gone)
    return got, t.size()


# ---------------------------------------------------------------- calls (small tables, with flags)


def _prepare_calls(s, c, seed):
    g = _gen(seed)
    n = c["n"]
    both = _distinct(n + n // 2 + 16, c["key"], seed)
    s.keys, absent = both[:n].clone(), both[n:].clone()
    s.vals = _values(s.keys, c["mapped"])
    s.queries = _queries(s.keys, absent, c["queries"], 0.6, g)
    s.gone = s.keys[torch.randperm(n, generator=g, device="cuda")[: max(1, n // 3)]].contiguous()
    s.new = torch.empty(n, dtype=torch.uint8, device="cuda")
    s.left = torch.empty(s.gone.numel(), dtype=torch.uint8, device="cuda")
    s.t = s.table()


def _run_calls(s):
    t = s.t
    t.insert(s.keys, s.vals, flags=s.new)
    got = t.find(s.queries) if s.case["mapped"] else t.contains(s.queries)
    t.erase(s.gone, flags=s.left)
    after = t.contains(s.queries)
    t.clear()
    return s.new, got, s.left, after


# ---------------------------------------------------------------- churn


def _prepare_churn(s, c, seed):
    g = _gen(seed)
    held = int(c["capacity"] * c["load"])
    universe = 1 << max(20, int(held * 1.3).bit_length())
    salt = (int(seed) * 0x2545F491) & ((1 << 40) - 1)
    s.t = s.table()
    for lo in range(0, held, 1 << 24):
        ids = torch.arange(lo, min(held, lo + (1 << 24)), device="cuda", dtype=torch.int64)
        keys = _mix64(ids + (salt << 20))
        s.t.insert(keys, _values(keys, c["mapped"]))
    # popular ranks are scattered over the ids, of which the first `held` are stored
    ids = (_zipf(c["batch"], universe, c["exponent"], g) * 0x9E3779B1 + 12345) & (universe - 1)
    s.batch = _mix64(ids + (salt << 20))
    s.vals = _values(s.batch, c["mapped"])
    new = torch.unique(ids[ids >= held])
    s.gone = _mix64(new[torch.randperm(new.numel(), generator=g, device="cuda")] + (salt << 20))


def _run_churn(s):
    t = s.t
    before = t.find(s.batch) if s.case["mapped"] else t.contains(s.batch)
    t.insert(s.batch, s.vals)
    size = t.size()
    after = t.contains(s.batch)
    t.erase(s.gone)
    return before, size, after, t.size()


# ---------------------------------------------------------------- hashed


def _spatial_hash(keys):
    """The usual spatial hash of three signed 16-bit coordinates packed into a word."""
    x, y, z = (((keys >> (16 * a)) & 0xFFFF) for a in range(3))
    x, y, z = (torch.where(v >= 32768, v - 65536, v) for v in (x, y, z))
    return (x * 73856093) ^ (y * 19349669) ^ (z * 83492791)


def _prepare_hashed(s, c, seed):
    g = _gen(seed)
    n = c["n"]
    extra = max(1024, n // 4)
    side = max(64, min(32768, int((24.0 * n) ** (1 / 3)) + 8))
    got = torch.empty(0, dtype=torch.int64, device="cuda")
    while got.numel() < n + extra:
        xyz = [torch.randint(-side, side, (int((n + extra) * 1.2) + 1024,), generator=g, device="cuda",
                             dtype=torch.int64) & 0xFFFF for _ in range(3)]
        got = torch.unique(torch.cat([got, xyz[0] | (xyz[1] << 16) | (xyz[2] << 32)]))
    got = got[torch.randperm(got.numel(), generator=g, device="cuda")]
    s.keys, absent = got[:n].clone(), got[n:n + extra].clone()
    s.vals = _values(s.keys, c["mapped"])
    s.queries = _queries(s.keys, absent, c["queries"], c["hits"], g)
    s.gone = s.keys[: n // 3].clone()
    s.hashes, s.hq, s.hgone = _spatial_hash(s.keys), _spatial_hash(s.queries), _spatial_hash(s.gone)
    s.t = s.table(custom_hash=True)


def _run_hashed(s):
    t = s.t
    t.clear()
    t.insert(s.keys, s.vals, hashes=s.hashes)
    got = t.find(s.queries, hashes=s.hq) if s.case["mapped"] else t.contains(s.queries, hashes=s.hq)
    t.erase(s.gone, hashes=s.hgone)
    return got, t.size()


# ---------------------------------------------------------------- merge


def _prepare_merge(s, c, seed):
    g = _gen(seed)
    n = c["n"]
    both = _distinct(n + n // 2 + 16, c["key"], seed)
    keys, absent = both[:n].clone(), both[n:].clone()
    s.source = s.table()
    s.source.insert(keys, _values(keys, c["mapped"]))
    s.dest = s.table(capacity=c["into"])
    s.queries = _queries(keys, absent, c["queries"], 0.7, g)


def _run_merge(s):
    s.dest.clear()
    keys, vals = s.source.range_copy()
    s.dest.insert(keys, vals)
    got = s.dest.find(s.queries) if s.case["mapped"] else s.dest.contains(s.queries)
    return got, keys.numel()


# ---------------------------------------------------------------- batch


def _batch_counts(c):
    rng = np.random.default_rng(c["tables"])
    k = np.exp(rng.normal(math.log(c["median"]), 1.5, size=c["tables"]))
    return np.clip(np.round(k), 64, 128 * c["median"]).astype(np.int64)


def _prepare_batch(s, c, seed):
    g = _gen(seed)
    counts = _batch_counts(c)
    caps = 2 ** np.ceil(np.log2(2 * counts)).astype(np.int64)
    s.b = s.own(sg.table_batch.createDeviceObjects(caps, key=c["key"], mapped=c["mapped"] or None),
                sg.table_batch.destroyDeviceObjects)
    off = np.concatenate([[0], np.cumsum(counts)])
    n = int(off[-1])
    s.offsets = torch.from_numpy(off).cuda()
    both = _distinct(2 * n, c["key"], seed)
    s.keys, fresh = both[:n].clone(), both[n:].clone()
    s.vals = _values(s.keys, c["mapped"])
    # a table's queries: its own keys or keys that no table holds
    first = torch.repeat_interleave(s.offsets[:-1], s.offsets[1:] - s.offsets[:-1])
    size = torch.repeat_interleave(s.offsets[1:] - s.offsets[:-1], s.offsets[1:] - s.offsets[:-1])
    own = first + (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * size).long().clamp_max(size - 1)
    hit = torch.rand(n, generator=g, device="cuda") < c["hits"]
    s.queries = torch.where(hit, s.keys[own], fresh).contiguous()


def _run_batch(s):
    s.b.clear()
    s.b.insert(s.keys, s.offsets, s.vals)
    got = s.b.find(s.queries, s.offsets) if s.case["mapped"] else s.b.contains(s.queries, s.offsets)
    return got, s.b.sizes()


# ---------------------------------------------------------------- worklist


def _prepare_worklist(s, c, seed):
    g = _gen(seed)
    n = c["n"]
    s.ids = torch.arange(n, device="cuda")  # each thread's candidate id
    s.pred = (torch.rand(n, generator=g, device="cuda") < c["share"]).to(torch.uint8)
    s.pushed = torch.empty(n, dtype=torch.uint8, device="cuda")
    s.bits = torch.randint(-(1 << 31), 1 << 31, ((c["bits"] + 31) // 32,), generator=g, device="cuda",
                           dtype=torch.int32)
    s.v = s.own(sg.vector.createDeviceObject(n, 8), sg.vector.destroyDeviceObject)


def _run_worklist(s):
    c = s.case
    s.v.clear()
    s.v.push_back(s.ids, s.pred, flags=s.pushed)
    occupied = sg.bitset_count(s.bits, c["bits"])
    todo = s.v.data()
    marked = torch.zeros(c["n"], dtype=torch.uint8, device="cuda").index_fill_(0, todo, 1)
    return s.pushed, marked, occupied, todo.numel()


# ---------------------------------------------------------------- queue


def _prepare_queue(s, c, seed):
    g = _gen(seed)
    n = c["n"]
    half = n // 2
    s.d = s.own(sg.deque.createDeviceObject(4 * n, 8), sg.deque.destroyDeviceObject)
    # the queue starts with as many ids as two passes pop, in a fixed order
    held = torch.randperm(4 * n, generator=g, device="cuda")[: 2 * half].sort().values
    s.d.push_front(held)
    # as many pushes as pops, mixed; a pass pops what an earlier one pushed
    s.push = (torch.randperm(2 * half, generator=g, device="cuda") < half).to(torch.uint8)
    s.ids = torch.randperm(4 * n, generator=g, device="cuda")[: 2 * half].sort().values
    # an element that pushed popped nothing (0): it marks a place of its own behind the ids
    s.own_place = torch.where(s.push != 0, 4 * n + torch.arange(2 * half, device="cuda"), 0)


def _run_queue(s):
    popped, ok = s.d.ops(s.push, s.ids)
    seen = torch.zeros(5 * s.case["n"], dtype=torch.uint8, device="cuda")
    seen.index_fill_(0, popped.add_(s.own_place), 1)
    return seen, ok, s.d.size()


# ---------------------------------------------------------------- served


def _prepare_served(s, c, seed):
    g = _gen(seed)
    rng = np.random.default_rng(c["requests"])
    s.server = s.own(sg_server.server(key="u64", mapped="u64", budget_bytes=16 << 30),
                     lambda srv: srv.close())
    lo, hi = math.log(c["cap_least"]), math.log(c["cap_most"])
    for t in range(c["tables"]):
        s.server.admit(t, int(math.exp(rng.uniform(lo, hi))))
    lo, hi = math.log(c["least"]), math.log(c["most"])
    asked = [(int(rng.integers(0, c["tables"])),
              int(rng.choice([sg_server.INSERT, sg_server.FIND, sg_server.ERASE], p=[0.4, 0.5, 0.1])),
              int(math.exp(rng.uniform(lo, hi)))) for _ in range(c["requests"])]
    # the finds' results lie one after another in two arrays
    s.vals, s.found = s.server.new_outputs(sum(n for _, op, n in asked if op == sg_server.FIND))
    s.items, at = [], 0
    for t, op, n in asked:
        keys = _mix64(_zipf(n, 1 << 30, 0.99, g) + _word((t << 40) + (int(seed) * 0x9E3779B97F4A7C15)))
        vals = _values(keys, "u64") if op == sg_server.INSERT else None
        if op == sg_server.FIND:
            s.items.append((t, op, keys, None, s.vals[at: at + n], s.found[at: at + n]))
            at += n
        else:
            s.items.append((t, op, keys, vals, None, None))


def _run_served(s):
    s.server.submit_many(s.items)
    s.server.drain()
    return s.vals, s.found, [s.server.table_size(t) for t in range(min(32, s.case["tables"]))]


# ---------------------------------------------------------------- the four functions

_PREPARE = {"step": _prepare_step, "calls": _prepare_calls, "churn": _prepare_churn, "hashed": _prepare_hashed,
            "merge": _prepare_merge, "batch": _prepare_batch, "worklist": _prepare_worklist, "queue": _prepare_queue,
            "served": _prepare_served}
_RUN = {"step": _run_step, "calls": _run_calls, "churn": _run_churn, "hashed": _run_hashed, "merge": _run_merge,
        "batch": _run_batch, "worklist": _run_worklist, "queue": _run_queue, "served": _run_served}


def prepare(case, seed):
    s = State(case)
    _PREPARE[case["family"]](s, case, int(seed))
    torch.cuda.synchronize()
    return s


def run(state):
    return _RUN[state.case["family"]](state)


def _storage(key, mapped, capacity):
    """Bytes of the slots of a table: the reference's geometry."""
    kind = sg.KINDS[(key, mapped or None)]
    g = sg.geometry_for(kind, int(capacity))
    return g.max_size * g.slot_bytes


def work(case):
    """Bytes that a pass cannot do without: inputs and outputs once; a cleared table's slots written once, a copied
    table's read once; one 32-byte sector read for each key looked up, inserted or erased, and one written for
    each key that changes a slot.  There is no arithmetic to speak of."""
    c, f = case, case["family"]
    sector = 32
    k, m = KEY_BYTES.get(c.get("key"), 8), MAPPED_BYTES.get(c.get("mapped"), 0)
    if f == "step":
        e = max(1, int(c["n"] * c["erase"]))
        b = _storage(c["key"], c["mapped"], c["capacity"])
        b += c["n"] * (k + m + 2 * sector) + c["queries"] * (k + m + 1 + sector) + e * (k + 2 * sector)
    elif f == "calls":
        b = _storage(c["key"], c["mapped"], c["capacity"])
        b += c["n"] * (k + m + 1 + 2 * sector) + c["queries"] * (2 * k + m + 2 + 2 * sector)
        b += max(1, c["n"] // 3) * (k + 1 + 2 * sector)
    elif f == "churn":
        b = c["batch"] * (3 * k + 2 * m + 2 + 3 * sector)
    elif f == "hashed":
        b = _storage(c["key"], c["mapped"], c["capacity"])
        b += c["n"] * (k + 8 + m + 2 * sector) + c["queries"] * (k + 8 + m + 1 + sector)
        b += c["n"] // 3 * (k + 8 + 2 * sector)
    elif f == "merge":
        b = _storage(c["key"], c["mapped"], c["capacity"]) + _storage(c["key"], c["mapped"], c["into"])
        b += c["n"] * (2 * (k + m) + 2 * sector) + c["queries"] * (k + m + 1 + sector)
    elif f == "batch":
        counts = _batch_counts(c)
        caps = 2 ** np.ceil(np.log2(2 * counts)).astype(np.int64)
        n = int(counts.sum())
        b = 3 * sum(_storage(c["key"], c["mapped"], x) * int(y) for x, y in zip(*np.unique(caps, return_counts=True)))
        b += n * (k + m) + n * (k + m + 1)
    elif f == "worklist":
        n, p = c["n"], int(c["n"] * c["share"])
        b = n * 2 + p * 16 + c["bits"] // 8 + p * 16 + n + p
    elif f == "queue":
        n = c["n"]
        b = n * (1 + 1 + 8 + 8 + 4) + 4 * n
    else:
        mean = (c["most"] - c["least"]) / math.log(c["most"] / c["least"])
        b = int(c["requests"] * mean * (8 + 8 + 2 * sector))
    return {"bytes": int(b), "flops": 0}
