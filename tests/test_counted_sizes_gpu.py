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
