"""Leaf rows rewritten in place: from one new key a leaf to as many as fit it,
before, between and behind its keys, and from one deleted key to all of them,
by the general path's kernels and the small batches'."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump, run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("touch_sort", [1, 2])
@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 7])
def test_leaf_rows(gpu, count, touch_sort):
    rng = np.random.default_rng(count)
    leaves = 90
    keys = np.arange(1, 24 * leaves + 1).astype(np.uint64) * np.uint64(1 << 33)
    t = E.BTree(max_keys=1 << 15, max_batch=1 << 12)
    t.set_option(E.OPT_TOUCH_SORT, touch_sort)
    t.bulk_build(dev(keys), dev(O.value_of(keys)))
    want = dict(zip(keys.tolist(), O.value_of(keys).tolist()))
    new = []
    for b in range(leaves):  # at the leaf's start, its end, or anywhere in it
        lo, hi = int(keys[24 * b]), int(keys[24 * b + 23])
        if b % 3 == 0:
            new += [lo + 1 + i for i in range(count)]
        elif b % 3 == 1:
            new += [hi + 1 + i for i in range(count)]
        else:
            new += (np.unique(rng.integers(lo + 1, hi, 40, dtype=np.int64))[:count] | 1).tolist()
    new = np.unique(np.array(new, dtype=np.uint64))
    rng.shuffle(new)
    run_batch(t, new, O.value_of(new), np.zeros(new.size, np.uint8), E.MODE_SORTED | E.MODE_MERGE_ENGINE)
    want.update(zip(new.tolist(), O.value_of(new).tolist()))
    assert t.leaf_sizes().size == leaves  # nothing split

    gk, gv = dump(t)
    assert gk.tolist() == sorted(want) and gv.tolist() == [want[k] for k in sorted(want)]
    # `count` keys of every leaf deleted, whole leaves among them
    edge = np.concatenate([[0], np.cumsum(t.leaf_sizes())]).astype(np.int64)
    gone = []
    for b in range(leaves):
        a, e = edge[b], edge[b + 1]
        gone += gk[a:e].tolist() if b % 9 == 4 else gk[a + rng.permutation(e - a)[:count]].tolist()
    gone = np.array(gone, np.uint64)
    rng.shuffle(gone)
    run_batch(t, gone, O.value_of(gone), np.full(gone.size, E.OP_DELETE, np.uint8), E.MODE_SORTED | E.MODE_MERGE_ENGINE)
    for k in gone.tolist():
        del want[k]
    gk, gv = dump(t)
    assert gk.tolist() == sorted(want) and gv.tolist() == [want[k] for k in sorted(want)]
    # every stored key is found by its fingerprint, no deleted one
    ov, os_ = run_batch(t, np.concatenate([gk, gone]), np.zeros(gk.size + gone.size, np.uint64),
                        np.full(gk.size + gone.size, E.OP_GET, np.uint8), E.MODE_SORTED | E.MODE_MERGE_ENGINE)[:2]
    assert (ov[:gk.size] == gv).all() and not os_[gk.size:].any() and os_[:gk.size].all()
