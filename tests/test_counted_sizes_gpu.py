"""Bulk calls of tables that keep the reference's excess list, at the sizes where their launches change: one key,
a warp and its neighbours, a block, the blocks of a cluster, the last call that runs as one cluster and the first
that runs as three launches.  Outcomes per key, size() and the keys in excess slots equal the oracle's
(src/stdgpu/impl/unordered_base_detail.cuh:708-913, 958-1043, one thread in input order)."""

import numpy as np
import pytest

import oracle as O

from gpu_util import per_key_success
from test_unordered_gpu import Table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 2047, 2049, 4095, 4096, 4097, 8200, 30001])
@pytest.mark.parametrize("kind", [O.SET_U32, O.MAP_U64_U32, O.MAP_U32_U32])
def test_insert_and_erase_equal_the_oracle(kind, n):
    rng = np.random.default_rng(1000 * kind + n)
    t, P = Table(kind, 3 * n + 5), O.PortTable(kind, 3 * n + 5)
    kd, vd = O.KEY_DTYPE[kind], O.VAL_DTYPE[kind]
    top = np.iinfo(kd).max
    for call in range(3):
        # copies of keys, keys stored by an earlier call, and the two keys that are kept out of the groups
        keys = rng.integers(0, 2 * n + 3, size=n).astype(kd) * kd(2654435761)
        if n > 2:
            keys[rng.integers(0, n, size=2)] = [top, top - kd(1)]
        vals = (keys ^ kd(77)).astype(vd) if vd is not None else None
        assert per_key_success(keys, t.insert(keys, vals)) == per_key_success(keys, P.insert(keys, vals, flags=True))
        assert t.size() == P.size() and t.t.excess_used() == P.excess_used()
        gone = keys[rng.permutation(n)[: (n + 1) // 2]]
        assert per_key_success(gone, t.erase(gone)) == per_key_success(gone, P.erase(gone, flags=True))
        assert t.size() == P.size() and t.t.excess_used() == P.excess_used()
    assert t.valid()
    order = np.argsort(t.range()[0])
    porder = np.argsort(P.range()[0])
    assert np.array_equal(t.range()[0][order], P.range()[0][porder])
    if vd is not None:
        assert np.array_equal(t.range()[1][order], P.range()[1][porder])
    t.t.clear()
    assert t.size() == 0 and t.t.excess_used() == 0 and t.valid()
    t.close()
    P.close()


@pytest.mark.parametrize("n", [1, 33, 1000, 70001])
@pytest.mark.parametrize("kind", [O.MAP_U64_U32, O.MAP_U32_U64, O.MAP_U64_U64])
def test_absent_keys_read_back_as_zero(kind, n):
    """find() returns 0 for absent keys whatever its output memory held, the two out-of-band keys included; the C
    entry point sg_unordered_find leaves them alone."""
    import torch

    from gpu_util import dev, host
    from stdgpu_gb300 import _native as N

    kd, vd = O.KEY_DTYPE[kind], O.VAL_DTYPE[kind]
    t = Table(kind, 4 * n)
    keys = (np.arange(n).astype(kd) + kd(1)) * kd(2654435761)
    vals = (keys >> kd(3)).astype(vd)
    t.insert(keys, vals)
    top = np.iinfo(kd).max
    q = np.concatenate([keys[::2], ~keys, np.array([top, top - kd(1)], kd)])
    stored = np.isin(q, keys)
    want = np.where(stored, (q >> kd(3)).astype(vd), vd(0)).astype(vd)
    del_me = torch.full((4 * q.size,), -1, dtype=torch.int64, device="cuda")  # what the allocator hands out next
    del del_me
    got, found = t.find(q)
    assert np.array_equal(found, stored.astype(np.uint8)) and np.array_equal(got, want)
    out = dev(np.full(q.size, 5, vd))
    flag = torch.empty(q.size, dtype=torch.uint8, device="cuda")
    N.check(N.load().sg_unordered_find(t.t._h, dev(q).data_ptr(), q.size, out.data_ptr(), flag.data_ptr(), None), "find")
    torch.cuda.synchronize()
    assert np.array_equal(host(out, vd), np.where(stored, want, vd(5)))
    t.close()
