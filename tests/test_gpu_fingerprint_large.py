"""Leaf fingerprints in the kernels that only large calls reach: the plain lookups
by warps (65,536 requests and more) and the locates of a batch's written keys
(every batch size under BT_OPT_TOUCH_SORT 1 and 0), on leaves whose every slot has
the key's fingerprint and after every kind of writer, against a dictionary."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, empty_u64, empty_u8, host_u64, host_u8, run_batch
from tests.test_gpu_fingerprint import fp

pytestmark = pytest.mark.gpu
MERGE = E.MODE_SORTED | E.MODE_MERGE_ENGINE


def answers(d, q):
    st = np.array([k in d for k in q.tolist()], np.uint8)
    return np.array([d.get(k, 0) for k in q.tolist()], np.uint64), st


def check(t, d, q):
    # tiled to the smallest sizes of the warp form; its last warp is whole or has one request
    q = np.concatenate([q, [np.uint64(E.KEY_MAX)]])
    wv, ws = answers(d, q)
    ws[-1] = E.ST_REJECTED
    t.set_descent(False)
    for n in (65_536, 65_537):
        at = np.arange(n) % q.size
        ov, os_ = empty_u64(n), empty_u8(n)
        t.search(dev(q[at]), ov, os_)
        assert (host_u8(os_) == ws[at]).all() and (host_u64(ov) == wv[at]).all(), n


@pytest.mark.parametrize("same", [False, True])
@pytest.mark.parametrize("touch_sort", [2, 1, 0])
def test_writers_in_turn(gpu, same, touch_sort, tmp_path):
    rng = np.random.default_rng(2001)
    pool = np.unique(rng.integers(0, 1 << 63, 1_200_000).astype(np.uint64))
    rng.shuffle(pool)
    pool = pool[fp(pool) == 77] if same else pool[:4_500]
    keys, fresh, never = np.sort(pool[:1_500]), pool[1_500:3_500], pool[3_500:]
    t = E.BTree(max_keys=1 << 16, max_batch=1 << 17)
    t.set_option(E.OPT_TOUCH_SORT, touch_sort)
    t.bulk_build(dev(keys), dev(O.value_of(keys)))
    d = dict(zip(keys.tolist(), O.value_of(keys).tolist()))
    q = np.concatenate([keys, fresh, never[:500]])
    check(t, d, q)

    def step(tree, i, mode):
        # fresh keys in (leaves split), stored ones updated and deleted, absent ones deleted
        ins = fresh[i * 250:(i + 1) * 250]
        stored = np.array(sorted(d), np.uint64)
        part = rng.permutation(stored.size)
        upd, gone = stored[part[:200]], np.concatenate([stored[part[200:320]], never[i * 20:i * 20 + 20]])
        rk = np.concatenate([ins, upd, gone])
        rv = O.value_of(rk) ^ np.uint64(i + 1)
        ro = np.concatenate([np.full(ins.size + upd.size, E.OP_INSERT), np.full(gone.size, E.OP_DELETE)]).astype(np.uint8)
        if i % 2:  # as a batch above the small ones' limit: the same writes among GETs
            g = np.tile(never, 66_000 // never.size + 1)[:66_000]
            rk, rv = np.concatenate([rk, g]), np.concatenate([rv, g])
            ro = np.concatenate([ro, np.full(g.size, E.OP_GET, np.uint8)])
        at = rng.permutation(rk.size)
        if mode != E.MODE_STM:
            wv, ws = answers(d, rk)  # (the GETs ask for keys that are never there)
        got = run_batch(tree, rk[at], rv[at], ro[at], mode)
        if mode != E.MODE_STM:
            assert (got[1] == ws[at]).all() and (got[0] == wv[at]).all(), i
        d.update(zip(rk[:ins.size + upd.size].tolist(), rv[:ins.size + upd.size].tolist()))
        for k in gone.tolist():
            d.pop(k, None)
        check(tree, d, q)

    for i, mode in enumerate((MERGE, MERGE, E.MODE_SORTED, E.MODE_STM, MERGE, E.MODE_SORTED)):
        step(t, i, mode)
    path = str(tmp_path / "pool")
    t.save_image(path)
    u = E.BTree(max_keys=1 << 16, max_batch=1 << 17)
    u.set_option(E.OPT_TOUCH_SORT, touch_sort)
    u.load_image(path)
    check(u, d, q)
    for i, mode in ((6, MERGE), (7, MERGE)):
        step(u, i, mode)
