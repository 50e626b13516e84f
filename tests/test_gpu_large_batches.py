"""Batches above the small ones' 65,536 requests in flight together: host batches
chained one beside the other's tree part, packed values, values read in place,
several batches of a call, small batches and other calls between them, the
deferred merge under a call on another stream.  The write share changes from
batch to batch, so that the cluster write part, the sample sort and the radix
sort follow one another.  Every answer, the contents and the tree's shape against
the oracle run in call order."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump, empty_u64, empty_u8, host_u64, host_u8

pytestmark = pytest.mark.gpu
MERGE = E.MODE_SORTED | E.MODE_MERGE_ENGINE
SHARES = [99, 50, 0, 95, 100, 80, 99, 20]


def requests(seed, keys, n, pct, deletes=0.0):
    rng = np.random.default_rng(seed)
    rk, rv, ro = O.gen_requests("uniform", seed, keys, n, pct)
    hot = rng.integers(0, n, n // 16)  # repeated keys in the batch
    rk[hot] = rk[rng.integers(0, 200, hot.size)]
    ro = ro.copy()
    ro[rng.random(n) < deletes] = E.OP_DELETE
    return rk, rv, ro


def distinct(rk, rv, ro):
    sel = np.sort(np.unique(rk, return_index=True)[1])  # STM answers that do not depend on an order
    return rk[sel], rv[sel], ro[sel]


def host_buffers(rk, rv, ro):
    import torch

    return [torch.from_numpy(x).pin_memory() for x in
            (rk.view(np.int64).copy(), rv.view(np.int64).copy(), ro.copy(), np.zeros(rk.size, np.int64),
             np.zeros(rk.size, np.uint8))]


def same_tree(t, o, stm=False):
    t.sync()
    gk, gv = dump(t)
    ok, ov = o.dump()
    assert (gk == ok).all() and (gv == ov).all()
    if not stm:
        assert (t.leaf_sizes() == o.leaf_sizes()).all() and (t.level_counts() == o.level_counts()).all()
    assert t.stats()["error"] == 0


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("touch_sort", [2, 1, 0])
@pytest.mark.parametrize("in_place", [0, 1])
def test_host_batches_chain_beside_other_calls(gpu, learned, touch_sort, in_place):
    keys = O.gen_keys("uniform", 1701, 150_000)
    t = E.BTree(max_keys=1 << 22, max_batch=1 << 17)
    t.set_option(E.OPT_TOUCH_SORT, touch_sort)
    t.set_option(E.OPT_HOST_VALUES_IN_PLACE, in_place)
    t.bulk_build(dev(keys), dev(O.value_of(keys)))
    o = O.OracleTree()
    o.bulk_build(keys, O.value_of(keys))
    if learned:
        t.retrain()
        t.set_descent(True)
    plan = ["host", "packed", "host", "packed", "packed", "host", "dev", "host", "packed", "search", "host", "small",
            "packed", "many", "host", "host", "off", "host", "packed", "on", "packed", "stm", "host", "packed", "small",
            "host"]
    keep, checks, inflight, stm = [], [], [], False
    for i, what in enumerate(plan):
        if what in ("off", "on"):
            t.set_option(E.OPT_HOST_FRONT_OVERLAP, int(what == "on"))
            continue
        n = 9_999 if what == "small" else 66_001 + 9_973 * (i % 6)
        r = requests(1710 + i, keys, n, SHARES[i % len(SHARES)], 0.05 if i % 3 == 1 else 0.0)
        if what == "stm":
            r = distinct(*r)
            stm = True
            ex = o.execute_serial(*r)
        else:
            if what == "search":
                r = (r[0], r[1], np.full(n, E.OP_GET, np.uint8))
            ex = o.execute_merged(*r, engine=O.ENGINE_MERGE)
        if what in ("dev", "search", "many"):
            d, out = tuple(dev(x) for x in r), (empty_u64(n), empty_u8(n))
            if what == "dev":
                t.execute(*d, *out, mode=MERGE)
            elif what == "search":
                t.search(d[0], *out)
            else:  # this batch, a small one and a third of another share
                more = [requests(1810 + j, keys, m, p) for j, (m, p) in enumerate([(3_001, 60), (80_003, 99)])]
                exs = [ex] + [o.execute_merged(*m, engine=O.ENGINE_MERGE) for m in more]
                bs = [d] + [tuple(dev(x) for x in m) for m in more]
                outs = [out] + [(empty_u64(m[0].size), empty_u8(m[0].size)) for m in more]
                t.execute_many(bs, outs, mode=MERGE)
                keep.append((bs, outs))
                checks += [(i, e, *x, False) for e, x in zip(exs[1:], outs[1:])]
            keep.append(d)
            checks.append((i, ex, *out, False))
            continue
        hb = host_buffers(*r)
        if what == "packed":
            import torch

            ins = torch.from_numpy(r[1][r[2] == E.OP_INSERT].view(np.int64).copy()).pin_memory()
            hb.append(ins)
            inflight.append(t.submit_host_packed(hb[0], hb[2], ins, hb[3], hb[4], mode=MERGE))
        else:
            inflight.append(t.submit_host(*hb, mode=E.MODE_STM if what == "stm" else MERGE))
        keep.append(hb)
        checks.append((i, ex, hb[3], hb[4], True))
        while len(inflight) > 2:
            t.wait_host(inflight.pop(0))
    for tk in inflight:
        t.wait_host(tk)
    t.sync()
    for i, (ov, os_), a, s, host in checks:
        ga, gs = (a.numpy().view(np.uint64), s.numpy()) if host else (host_u64(a), host_u8(s))
        assert (gs == os_).all() and (ga == ov).all(), (i, plan[i])
    same_tree(t, o, stm)


def test_refused_packed_batch_between_chained_ones(gpu):
    # a value count that does not match the INSERTs: that batch alone is refused
    import torch

    keys = O.gen_keys("uniform", 1851, 100_000)
    t = E.BTree(max_keys=1 << 20, max_batch=1 << 17)
    t.bulk_build(dev(keys), dev(O.value_of(keys)))
    o = O.OracleTree()
    o.bulk_build(keys, O.value_of(keys))
    work = []
    for i in range(5):
        r = requests(1860 + i, keys, 70_000 + i, 50)
        hb = host_buffers(*r)
        ins = torch.from_numpy(r[1][r[2] == E.OP_INSERT].view(np.int64).copy()).pin_memory()
        if i == 2:
            ins, ex = ins[:-1], None
        else:
            ex = o.execute_merged(*r, engine=O.ENGINE_MERGE)
        work.append((t.submit_host_packed(hb[0], hb[2], ins, hb[3], hb[4], mode=MERGE), hb, ins, ex))
    for i, (tk, hb, _, ex) in enumerate(work):
        if ex is None:
            with pytest.raises(E.BTError):
                t.wait_host(tk)
            assert (hb[4].numpy() == E.ST_REJECTED).all()
            continue
        t.wait_host(tk)
        assert (hb[4].numpy() == ex[1]).all() and (hb[3].numpy().view(np.uint64) == ex[0]).all(), i
    same_tree(t, o)


@pytest.mark.parametrize("touch_sort", [2, 1, 0])
def test_calls_after_a_deferred_batch(gpu, touch_sort):
    # the answers are waited for; the leaf and inner merge may still run when a
    # call on another stream follows
    import torch

    keys = O.gen_keys("gamma", 1901, 100_000)
    t = E.BTree(max_keys=1 << 22, max_batch=1 << 18)
    t.set_option(E.OPT_TOUCH_SORT, touch_sort)
    t.bulk_build(dev(keys), dev(O.value_of(keys)))
    o = O.OracleTree()
    o.bulk_build(keys, O.value_of(keys))
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    rng = np.random.default_rng(1902)
    for b, n in enumerate([200_000, 70_000, 250_000, 70_001, 131_072]):
        new = rng.integers(1, 2**63, n, dtype=np.uint64)
        if b == 3:  # few writes: the cluster's form
            new[1_500:] = rng.choice(keys, n - 1_500)
        op = np.full(n, E.OP_INSERT, np.uint8)
        if b == 3:
            op[1_500:] = E.OP_GET
        rv = new ^ np.uint64(b + 7)
        o.execute_merged(new, rv, op, engine=O.ENGINE_MERGE)
        ins = op == E.OP_INSERT
        d, out = (dev(new), dev(rv), dev(op)), (empty_u64(n), empty_u8(n))
        qk, qv, qs = dev(new[ins]), empty_u64(int(ins.sum())), empty_u8(int(ins.sum()))
        torch.cuda.synchronize()
        t.execute(*d, *out, mode=MERGE, stream=s1)
        s1.synchronize()
        t.search(qk, qv, qs, stream=s2)
        lo, hi = dev(np.sort(new[ins])[:100]), dev(np.sort(new[ins])[:100])
        counts, k, _ = t.range(lo, hi, 2, stream=s2)
        s2.synchronize()
        assert (host_u8(qs) == E.ST_FOUND).all() and (host_u64(qv) == rv[ins]).all(), b
        assert (counts == 1).all() and (k[:, 0] == lo).all(), b
        assert t.size() == o.size()
    same_tree(t, o)


@pytest.mark.parametrize("touch_sort", [2, 1, 0])
@pytest.mark.parametrize("mode, engine", [(MERGE, O.ENGINE_MERGE), (E.MODE_SORTED, O.ENGINE_STM)])
@pytest.mark.parametrize("dist", ["uniform", "gamma"])
def test_batches_one_by_one(gpu, touch_sort, mode, engine, dist):
    # the general path at sizes that are no multiple of anything, both engines
    import torch

    keys = O.gen_keys(dist, 1951, 90_000)
    t = E.BTree(max_keys=1 << 21, max_batch=1 << 17)
    t.set_option(E.OPT_TOUCH_SORT, touch_sort)
    t.bulk_build(dev(keys), dev(O.value_of(keys)))
    o = O.OracleTree()
    o.bulk_build(keys, O.value_of(keys))
    for b, (n, pct, dfrac) in enumerate([(65_537, 95, 0.0), (90_001, 50, 0.1), (131_072, 5, 0.3), (70_001, 99, 0.01)]):
        r = requests(1960 + b, keys, n, pct, dfrac)
        ov, os_ = o.execute_merged(*r, engine=engine)
        out = (empty_u64(n), empty_u8(n))
        t.execute(*(dev(x) for x in r), *out, mode=mode)
        torch.cuda.synchronize()
        assert (host_u8(out[1]) == os_).all() and (host_u64(out[0]) == ov).all(), b
    same_tree(t, o, stm=engine == O.ENGINE_STM)
