"""Leaves that a batch cuts into many pieces (merge_leaf_kernel spreads the
pieces over the chip) against the oracle's merge engine: answers, contents and
the exact shape, for new keys below, between and above a leaf's old keys, beside
leaves that only take a key or two."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump, run_batch

pytestmark = pytest.mark.gpu
MERGE = E.MODE_SORTED | E.MODE_MERGE_ENGINE


@pytest.mark.parametrize("fill", [16, 24, 31])
@pytest.mark.parametrize("cnt", [1, 7, 8, 9, 31, 32, 49, 1000, 60_000])
def test_one_leaf_many_pieces(gpu, cnt, fill):
    step = np.uint64(1 << 40)
    keys = (np.arange(1, 5001).astype(np.uint64)) * step
    t = E.BTree(max_keys=1 << 21, max_batch=1 << 19, leaf_fill=fill, inner_fill=24)
    o = O.OracleTree(fill, 24)
    t.bulk_build(dev(keys), dev(O.value_of(keys)))
    o.bulk_build(keys, O.value_of(keys))
    rng = np.random.default_rng(cnt)
    parts = []
    for at in (0, 12, 2500, 2511, 5000):  # ahead of the first key, inside leaves, beyond the last key
        parts.append(keys[0] * np.uint64(at) + np.unique(rng.integers(1, 1 << 40, cnt).astype(np.uint64)))
    parts.append(keys[rng.integers(0, 5000, 600)] + np.uint64(5))  # leaves that only take a key or two
    rk = np.unique(np.concatenate(parts))
    rng.shuffle(rk)
    rv = O.value_of(rk)
    for b in range(2):  # the second batch cuts the pieces of the first
        ro = np.zeros(rk.size, np.uint8)
        ov, os_ = o.execute_merged(rk, rv, ro, O.ENGINE_MERGE)
        gv, gs = run_batch(t, rk, rv, ro, MERGE)
        assert (gs == os_).all() and (gv == ov).all(), b
        rk = np.unique(rk + np.uint64(1))
        rv = O.value_of(rk)
    gk, gvv = dump(t)
    ok, ovv = o.dump()
    assert gk.size == ok.size and (gk == ok).all() and (gvv == ovv).all()
    assert (t.leaf_sizes() == o.leaf_sizes()).all()
    assert (t.level_counts() == o.level_counts()).all()
    assert t.stats()["leaf_splits"] == o.stats()["leaf_splits"]
    assert t.stats()["error"] == 0
