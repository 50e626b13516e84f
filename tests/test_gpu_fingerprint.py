"""Leaf fingerprints (DevTree::fp): the plain and the learned lookups against a
dictionary where every slot of a leaf has the lookup's fingerprint, and after
every kind of writer (merge engine, STM, deletes, splits, a loaded pool image)
has changed the leaves, with the model fitted before and after."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, empty_u64, empty_u8, host_u64, host_u8, run_batch

pytestmark = pytest.mark.gpu
MERGE = E.MODE_SORTED | E.MODE_MERGE_ENGINE


def fp(k):
    with np.errstate(over="ignore"):
        h = k.astype(np.uint32) * np.uint32(0x9E3779B1) + (k >> np.uint64(32)).astype(np.uint32) * np.uint32(0x85EBCA77)
    return np.maximum(h >> np.uint32(24), 1)


def check(t, d, q):
    for learned in (False, True):
        t.set_descent(learned)
        ov, os_ = empty_u64(q.size), empty_u8(q.size)
        t.search(dev(q), ov, os_)
        want = np.array([d.get(k) is not None for k in q.tolist()], np.uint8)
        vals = np.array([d.get(k, 0) for k in q.tolist()], np.uint64)
        gs, gv = host_u8(os_), host_u64(ov)
        want[q == np.uint64(E.KEY_MAX)] = E.ST_REJECTED
        assert (gs == want).all() and (gv == vals).all(), learned


@pytest.mark.parametrize("n", [1, 31, 32, 33, 4097])
@pytest.mark.parametrize("same", [False, True])
def test_lookups_after_every_writer(gpu, n, same, tmp_path):
    rng = np.random.default_rng(17 + n)
    pool = np.unique(rng.integers(0, 1 << 63, 600_000).astype(np.uint64))
    rng.shuffle(pool)
    if same:  # one fingerprint everywhere: every slot is a candidate
        pool = pool[fp(pool) == 77]
    else:
        pool = pool[:2500]
    keys, fresh, never = np.sort(pool[:900]), pool[900:1600], pool[1600:]
    t = E.BTree(max_keys=1 << 16, max_batch=1 << 14)
    t.bulk_build(dev(keys), dev(O.value_of(keys)))
    d = dict(zip(keys.tolist(), O.value_of(keys).tolist()))
    t.retrain()
    q = np.concatenate([keys, fresh, never, [np.uint64(E.KEY_MAX)]])
    q = q[rng.integers(0, q.size, n)]
    check(t, d, q)
    for step, mode in enumerate((MERGE, E.MODE_SORTED, E.MODE_STM, MERGE)):
        ins = fresh[step * 175:(step + 1) * 175]
        gone = keys[step::9]
        rk = np.concatenate([ins, gone])
        ro = np.concatenate([np.full(ins.size, E.OP_INSERT), np.full(gone.size, E.OP_DELETE)]).astype(np.uint8)
        run_batch(t, rk, O.value_of(rk), ro, mode)
        d.update(zip(ins.tolist(), O.value_of(ins).tolist()))
        for k in gone.tolist():
            d.pop(k, None)
        check(t, d, q)  # the model is older than the leaves' splits
        if step == 1:
            t.refit()
            check(t, d, q)
    path = str(tmp_path / "pool")
    t.save_image(path)
    u = E.BTree(max_keys=1 << 16, max_batch=1 << 14)
    u.load_image(path)
    u.retrain()
    check(u, d, q)
    more = never[:300]
    run_batch(u, more, O.value_of(more), np.zeros(more.size, np.uint8), MERGE)
    d.update(zip(more.tolist(), O.value_of(more).tolist()))
    check(u, d, q)


def test_one_leaf_splits_more_often_than_its_byte_counts(gpu):
    # ascending fresh keys just above the leaf's low end split the same leaf
    # again and again: its split count saturates, and the fence decides
    keys = (np.arange(1, 2001).astype(np.uint64)) << np.uint64(40)
    t = E.BTree(max_keys=1 << 18, max_batch=1 << 12)
    t.bulk_build(dev(keys), dev(O.value_of(keys)))
    t.retrain()
    d = dict(zip(keys.tolist(), O.value_of(keys).tolist()))
    lo = int(keys[1000])
    for i in range(270):
        rk = np.array([lo + ((1 << 39) >> 0) - 40 * (i * 0 + 1) - 32 * i - j for j in range(32)], np.uint64)
        run_batch(t, rk, O.value_of(rk), np.zeros(32, np.uint8), MERGE)
        d.update(zip(rk.tolist(), O.value_of(rk).tolist()))
        if i in (0, 1, 200, 254, 255, 256, 269):
            q = np.concatenate([rk, rk + np.uint64(1 << 30), keys[990:1010], rk - np.uint64(1 << 30)])
            check(t, d, q)
            if i == 256:
                t.refit()
    check(t, d, np.array(list(d)[-9000:], np.uint64))
