"""Batches above the small ones' limit whose number of touched requests is not
that of the batch before, by which the host picks the sort and the form of the
write part: light before heavy and heavy before light, one by one, several in a
call and from host buffers, against the oracle (answers, contents, tree shape),
and their times."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump, empty_u64, empty_u8, host_u64, host_u8, run_batch

pytestmark = pytest.mark.gpu
MERGE = E.MODE_SORTED | E.MODE_MERGE_ENGINE


def requests(seed, keys, n, kind):
    rng = np.random.default_rng(seed)
    rk, rv, ro = O.gen_requests("uniform", seed, keys, n, {"light": 100, "few": 99, "half": 50}.get(kind, 0))
    if kind == "fresh":  # nothing but new keys: leaves split, inner nodes too
        rk = O.gen_keys("uniform", seed + 1, n)
        rv = O.value_of(rk)
    elif kind == "delete":
        rk = rng.choice(keys, n)
        ro = np.where(rng.random(n) < 0.7, E.OP_DELETE, E.OP_GET).astype(np.uint8)
    elif kind == "half":  # repeated keys with every op code in their runs, reserved key
        at = rng.integers(0, n, n // 8)
        rk[at] = rk[rng.integers(0, n, at.size) % 512]
        ro[rng.random(n) < 0.1] = E.OP_DELETE
        rk[:3], ro[3] = np.uint64(2**64 - 1), 7
    elif isinstance(kind, int):  # that many fresh keys among GETs of stored ones
        ro[:] = E.OP_GET
        rk = rng.choice(keys, n)
        rk[:kind] = O.gen_keys("uniform", seed + 1, kind)
        ro[:kind] = E.OP_INSERT
    return rk, rv, ro


def plan(n, beside):
    # the cluster's limit (cluster_write_limit): exactly that, and one more
    limit = min(n // 8, 20_480) if beside else 2_048
    return ["light", "fresh", "few", "delete", "light", "half", "few", limit + 1, "light", limit, "light", "few", "fresh"]


def same_tree(t, o):
    t.sync()
    gk, gv = dump(t)
    ok, ov = o.dump()
    assert (gk == ok).all() and (gv == ov).all()
    assert (t.leaf_sizes() == o.leaf_sizes()).all() and (t.level_counts() == o.level_counts()).all()
    assert t.stats()["error"] == 0 and t.size() == ok.size


@pytest.mark.parametrize("n", [65_537, 150_001, 1 << 19])
@pytest.mark.parametrize("call", ["each", "many", "host"])
@pytest.mark.parametrize("start", [200_000, 0])
def test_light_and_heavy_batches(gpu, n, call, start):
    import torch

    base = O.gen_keys("uniform", 1301, 200_000)
    t = E.BTree(max_keys=1 << 22, max_batch=1 << 19)
    o = O.OracleTree()
    if start:
        t.bulk_build(dev(base), dev(O.value_of(base)))
        o.bulk_build(base, O.value_of(base))
    kinds = plan(n, call != "each")
    reqs = [requests(1310 + 10 * i, base, n, k) for i, k in enumerate(kinds)]
    expect = [o.execute_merged(*r, engine=O.ENGINE_MERGE) for r in reqs]
    got = []
    if call == "each":
        for r in reqs:  # (waits: the hint is the batch before's)
            got.append(run_batch(t, *r, MERGE))
    elif call == "many":
        # a light one first: all of a call's batches are queued by its count
        got.append(run_batch(t, *reqs[0], MERGE))
        b = [tuple(dev(x) for x in r) for r in reqs[1:]]
        outs = [(empty_u64(n), empty_u8(n)) for _ in b]
        t.execute_many(b, outs, mode=MERGE)
        t.sync()
        got += [(host_u64(v), host_u8(s)) for v, s in outs]
    else:
        hb, tickets = [], []
        for i, (k, v, op) in enumerate(reqs):
            x = [torch.from_numpy(a.copy()).pin_memory() for a in (k.view(np.int64), v.view(np.int64), op)]
            x += [torch.zeros(n, dtype=torch.int64).pin_memory(), torch.zeros(n, dtype=torch.uint8).pin_memory()]
            hb.append(x)
            if i % 2 and (op <= E.OP_DELETE).all():  # the INSERTs' values only
                p = torch.from_numpy(v[op == E.OP_INSERT].view(np.int64).copy()).pin_memory()
                x.append(p)
                tickets.append(t.submit_host_packed(x[0], x[2], p, x[3], x[4], mode=MERGE))
            else:
                tickets.append(t.submit_host(*x[:5], mode=MERGE))
            if i >= 2:
                t.wait_host(tickets[i - 2])
        for tk in tickets[-2:]:
            t.wait_host(tk)
        got = [(x[3].numpy().view(np.uint64), x[4].numpy()) for x in hb]
    for i, ((gv, gs), (ov, os_)) in enumerate(zip(got, expect)):
        assert (gs == os_).all() and (gv == ov).all(), (i, kinds[i])
    same_tree(t, o)


def test_heavy_batch_that_does_not_fit(gpu):
    # the node pool is full: as the general path answers, and nothing is written
    n = 150_000
    base = O.gen_keys("uniform", 1401, 20_000)
    fresh = O.gen_keys("uniform", 1402, n)
    light = np.random.default_rng(1403).choice(base, n)
    res = []
    for touch in (2, 0):
        t = E.BTree(max_keys=1_000, max_batch=1 << 18)
        t.set_option(E.OPT_TOUCH_SORT, touch)
        t.bulk_build(dev(base), dev(O.value_of(base)))
        run_batch(t, light, light, np.full(n, E.OP_GET, np.uint8), MERGE)
        got = run_batch(t, fresh, O.value_of(fresh), np.full(n, E.OP_INSERT, np.uint8), MERGE)
        t.sync()
        res.append((*got, *dump(t)))
        assert (got[1] == E.ST_NO_CAPACITY).all() and t.size() == base.size and t.stats()["error"] != 0
    for a, b in zip(*res):
        assert (a == b).all()


def test_heavy_batches_cost_the_same_after_light_ones(gpu):
    # 2^20 INSERTs, then DELETEs of the same keys, behind one another and behind
    # light batches: a guess may cost the better sort, not four times the batch
    import torch

    n = 1 << 20
    keys = O.gen_keys("uniform", 1411, 1 << 21)
    t = E.BTree(max_keys=1 << 22, max_batch=n)
    t.bulk_build(dev(keys[n:]), dev(O.value_of(keys[n:])))
    k, light = dev(keys[:n]), dev(np.random.default_rng(1).choice(keys[n:], n))
    ops = {x: torch.full((n,), x, dtype=torch.uint8, device="cuda") for x in (E.OP_INSERT, E.OP_DELETE, E.OP_GET)}
    ov, os_ = empty_u64(n), empty_u8(n)
    s = torch.cuda.Stream()

    def ms(key, op):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda.synchronize()
        a.record(s)
        t.execute(key, key, ops[op], ov, os_, mode=MERGE, stream=s)
        t.sync(s)
        b.record(s)
        torch.cuda.synchronize()
        return a.elapsed_time(b)

    after = {"heavy": [], "light": []}
    for kind in after:
        for i in range(8):
            for op in (E.OP_INSERT, E.OP_DELETE):
                if kind == "light":
                    ms(light, E.OP_GET)
                after[kind].append(ms(k, op))
    steady, shifted = (np.median(after[x][4:]) for x in ("heavy", "light"))
    assert shifted < 1.6 * steady, (steady, shifted)


def test_two_handles_at_a_time(gpu):
    # two threads, each with a handle and a stream: light and heavy batches of both
    # meet on the device
    import threading

    import torch

    n, base = 130_000, O.gen_keys("uniform", 1421, 200_000)
    kinds = ["light", "fresh", "light", "delete", "few", "half", "light", 2_049, "light", "fresh"]
    reqs = [requests(1430 + 10 * i, base, n, k) for i, k in enumerate(kinds)]
    o = O.OracleTree()
    o.bulk_build(base, O.value_of(base))
    expect = [o.execute_merged(*r, engine=O.ENGINE_MERGE) for r in reqs]
    b = [tuple(dev(x) for x in r) for r in reqs]
    k, v = dev(base), dev(O.value_of(base))
    trees = [E.BTree(max_keys=1 << 21, max_batch=1 << 18) for _ in range(2)]
    outs = [[(empty_u64(n), empty_u8(n)) for _ in b] for _ in trees]
    torch.cuda.synchronize()
    errors = []

    def work(i):
        try:
            s = torch.cuda.Stream()
            for turn in range(4):
                trees[i].bulk_build(k, v, stream=s)
                if (i + turn) % 2:
                    for x, out in zip(b, outs[i]):
                        trees[i].execute(*x, *out, mode=MERGE, stream=s)
                else:
                    trees[i].execute_many(b, outs[i], mode=MERGE, stream=s)
                trees[i].sync(s)
                s.synchronize()
                for j, ((gv, gs), (ov, os_)) in enumerate(zip(outs[i], expect)):
                    assert (host_u8(gs) == os_).all() and (host_u64(gv) == ov).all(), (turn, j, kinds[j])
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    for t in trees:
        same_tree(t, o)
