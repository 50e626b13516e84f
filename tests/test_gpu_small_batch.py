"""Sorted batches of up to 65,536 requests (three launches: bt_small.cu) against
the oracle and against the general path (an explicit BT_OPT_TOUCH_SORT), at the
edges of the cluster sizes (128 requests per block), of the sort tiles (1024 to
4096 pairs) and of the path itself, for both insert engines."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump, run_batch

pytestmark = pytest.mark.gpu
MERGE = E.MODE_SORTED | E.MODE_MERGE_ENGINE
SIZES = [1, 2, 127, 128, 129, 1024, 1025, 2047, 4097, 16384, 16500, 40000, 65536, 65537]


def requests(rng, keys, n, mix):
    """Fresh and stored keys, repeated ones with every op code in their runs."""
    pool = np.concatenate([keys[rng.integers(0, keys.size, n)], rng.integers(0, 1 << 63, n).astype(np.uint64)])
    rk = pool[rng.integers(0, pool.size, n)]
    hot = rk[rng.integers(0, n, max(1, n // 100))]
    at = rng.integers(0, n, n // 6)
    rk[at] = hot[rng.integers(0, hot.size, at.size)]
    ro = np.full(n, E.OP_GET, np.uint8)
    w = rng.random(n) < mix
    ro[w] = np.where(rng.random(int(w.sum())) < 0.3, E.OP_DELETE, E.OP_INSERT)
    return rk, rng.integers(0, 1 << 62, n).astype(np.uint64), ro


@pytest.mark.parametrize("engine", ["merge", "stm"])
@pytest.mark.parametrize("mix", [0.0, 0.05, 0.5, 1.0])
@pytest.mark.parametrize("n", SIZES)
def test_small_batches_match_oracle(gpu, n, mix, engine):
    keys = O.gen_keys("uniform", 901, 30_000)
    vals = O.value_of(keys)
    t = E.BTree(max_keys=1 << 20, max_batch=1 << 17)
    t.bulk_build(dev(keys), dev(vals))
    o = O.OracleTree()
    o.bulk_build(keys, vals)
    rng = np.random.default_rng(int(1000 * mix) + n)
    for b in range(3):
        rk, rv, ro = requests(rng, keys, n, mix)
        ov, os_ = o.execute_merged(rk, rv, ro, engine=O.ENGINE_MERGE if engine == "merge" else O.ENGINE_STM)
        gv, gs = run_batch(t, rk, rv, ro, MERGE if engine == "merge" else E.MODE_SORTED)
        assert (gs == os_).all() and (gv == ov).all(), b
    gk, gvv = dump(t)
    ok, ovv = o.dump()
    assert gk.size == ok.size and (gk == ok).all() and (gvv == ovv).all()
    if engine == "merge":
        assert (t.leaf_sizes() == o.leaf_sizes()).all()
        assert (t.level_counts() == o.level_counts()).all()
    assert t.stats()["error"] == 0


@pytest.mark.parametrize("n", [5, 700, 9000, 65536])
def test_small_batches_from_empty_tree(gpu, n):
    t = E.BTree(max_keys=1 << 20, max_batch=1 << 16)
    o = O.OracleTree()
    rng = np.random.default_rng(n)
    for b in range(4):  # a root of one leaf, then growing levels
        rk = rng.integers(0, 1 << 63, n).astype(np.uint64)
        rv, ro = O.value_of(rk), np.zeros(n, np.uint8)
        ov, os_ = o.execute_merged(rk, rv, ro, engine=O.ENGINE_MERGE)
        gv, gs = run_batch(t, rk, rv, ro, MERGE)
        assert (gs == os_).all() and (gv == ov).all(), b
    assert (t.leaf_sizes() == o.leaf_sizes()).all()
    assert (t.level_counts() == o.level_counts()).all()


@pytest.mark.parametrize("n", [3, 300, 5000, 65536])
def test_small_batches_reserved_invalid_and_hot(gpu, n):
    # reserved keys, invalid op codes, one key in every request of a sort tile
    keys = O.gen_keys("uniform", 903, 20_000)
    vals = O.value_of(keys)
    rng = np.random.default_rng(n)
    got = []
    for opt in (2, 1):  # the small path, the general path
        t = E.BTree(max_keys=1 << 20, max_batch=1 << 16)
        t.set_option(E.OPT_TOUCH_SORT, opt)
        t.bulk_build(dev(keys), dev(vals))
        r = np.random.default_rng(n)
        for b in range(3):
            rk, rv, ro = requests(r, keys, n, 0.4)
            rk[r.random(n) < 0.05] = E.KEY_MAX
            ro[r.random(n) < 0.05] = 7
            if b:
                rk[n // 4:] = rk[0] if b == 1 else E.KEY_MAX
            got.append((b, *run_batch(t, rk, rv, ro, MERGE)))
        got.append((9, *dump(t)))
    half = len(got) // 2
    for x, y in zip(got[:half], got[half:]):
        assert x[1].size == y[1].size and (x[1] == y[1]).all() and (x[2] == y[2]).all(), x[0]


def test_small_batches_full_pool(gpu):
    # a pool too small for a batch's pieces: its new keys are answered kNoCapacity, nothing is inserted
    t = E.BTree(max_keys=1, max_batch=1 << 16)
    rng = np.random.default_rng(5)
    o = {}
    for b in range(6):
        rk = np.unique(rng.integers(0, 1 << 63, 30_000).astype(np.uint64))
        gv, gs = run_batch(t, rk, O.value_of(rk), np.zeros(rk.size, np.uint8), MERGE)
        assert (gs == E.ST_ABSENT).all() or (gs == E.ST_NO_CAPACITY).all()
        if gs[0] == E.ST_ABSENT:
            o.update(zip(rk.tolist(), O.value_of(rk).tolist()))
    gk, gv = dump(t)
    assert sorted(o) == gk.tolist() and [o[k] for k in gk.tolist()] == gv.tolist()
    assert t.stats()["error"] & 1


def test_small_and_large_batches_share_a_handle(gpu):
    # both paths in turn, in execute_many and through host buffers, one tree
    keys = O.gen_keys("uniform", 905, 50_000)
    vals = O.value_of(keys)
    t = E.BTree(max_keys=1 << 20, max_batch=1 << 17)
    t.bulk_build(dev(keys), dev(vals))
    o = O.OracleTree()
    o.bulk_build(keys, vals)
    rng = np.random.default_rng(7)
    for n in (100_000, 300, 70_000, 65_536, 5, 90_000):
        rk, rv, ro = requests(rng, keys, n, 0.2)
        ov, os_ = o.execute_merged(rk, rv, ro, engine=O.ENGINE_MERGE)
        gv, gs = run_batch(t, rk, rv, ro, MERGE)
        assert (gs == os_).all() and (gv == ov).all(), n
        rk, rv, ro = requests(rng, keys, n, 0.2)
        ov, os_ = o.execute_merged(rk, rv, ro, engine=O.ENGINE_MERGE)
        gv, gs = t.execute_host(rk, rv, ro, mode=MERGE)
        assert (gs == os_).all() and (gv == ov).all(), n
    import torch

    for sizes in ((400, 900, 30), (400, 80_000, 30)):
        batches = [requests(rng, keys, n, 0.2) for n in sizes]
        outs = [(torch.zeros(n, dtype=torch.int64, device="cuda"), torch.zeros(n, dtype=torch.uint8, device="cuda"))
                for n in sizes]
        t.execute_many([tuple(dev(x) for x in b) for b in batches], outs, mode=MERGE)
        torch.cuda.synchronize()
        for b, (ovt, ost) in zip(batches, outs):
            ov, os_ = o.execute_merged(*b, engine=O.ENGINE_MERGE)
            assert (ost.cpu().numpy() == os_).all() and (ovt.cpu().numpy().view(np.uint64) == ov).all()
    gk, gvv = dump(t)
    ok, ovv = o.dump()
    assert (gk == ok).all() and (gvv == ovv).all()
