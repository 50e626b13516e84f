"""Batches captured in a CUDA graph: the graph runs on the tree that is there
when it is replayed, and capturing leaves the handle as it was.  Without the
deferred write phase (OPT_ASYNC_WRITE 0) a batch is whole on its stream."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump, empty_u64, empty_u8, host_u64, host_u8, run_batch

pytestmark = pytest.mark.gpu
MERGE = E.MODE_SORTED | E.MODE_MERGE_ENGINE


class Captured:
    """One batch of n requests with buffers of its own; run() replays it."""

    def __init__(self, t, n, mode=MERGE):
        import torch

        self.bufs = empty_u64(n), empty_u64(n), empty_u8(n), empty_u64(n), empty_u8(n)
        self.graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(self.graph, capture_error_mode="thread_local"):
            t.execute(*self.bufs, mode=mode, stream=torch.cuda.current_stream())

    def run(self, keys, vals, ops):
        import torch

        for b, x in zip(self.bufs, (keys, vals, ops.astype(np.uint8))):
            b.copy_(dev(x))
        self.graph.replay()
        torch.cuda.synchronize()
        return host_u64(self.bufs[3]), host_u8(self.bufs[4])


def tree(max_keys=1 << 20, max_batch=1 << 17):
    t = E.BTree(max_keys=max_keys, max_batch=max_batch)
    t.set_option(E.OPT_ASYNC_WRITE, 0)
    return t


def inserts(seed, n):
    k = O.gen_keys("uniform", seed, n)
    return k, O.value_of(k), np.full(n, E.OP_INSERT, np.uint8)


@pytest.mark.parametrize("n", [3_000, 70_000])  # the small batches' kernels, the general path
def test_root_of_an_empty_tree(gpu, n):
    k, v, op = inserts(1201, n)
    t = tree()
    g = Captured(t, n)
    # captured only: this batch still has to make the root
    _, st = run_batch(t, k, v, op, MERGE)
    assert (st == E.ST_ABSENT).all() and t.size() == n
    # and the graph has to make one for a tree emptied after its capture
    t.bulk_build(empty_u64(0), empty_u64(0))
    _, st = g.run(k, v, op)
    assert (st == E.ST_ABSENT).all() and t.size() == n
    gk, gv = dump(t)
    o = np.argsort(k)
    assert (gk == k[o]).all() and (gv == v[o]).all()


@pytest.mark.parametrize("n", [3_000, 70_000, 131_072])
@pytest.mark.parametrize("mode, engine", [(MERGE, O.ENGINE_MERGE), (E.MODE_SORTED, O.ENGINE_STM)])
def test_replays_with_other_inputs(gpu, n, mode, engine):
    # every replay meets the tree and the counts of its own turn: fresh keys (many
    # tiles of new keys and segments, leaves that split), few writes, deletes
    keys, vals, _ = inserts(1211, 150_000)
    t = tree(max_keys=1 << 21)
    t.bulk_build(dev(keys), dev(vals))
    o = O.OracleTree()
    o.bulk_build(keys, vals)
    g = Captured(t, n, mode)
    rng = np.random.default_rng(1212)
    for turn, pct in enumerate([0, 20, 99, 0, 60]):
        rk, rv, ro = O.gen_requests("uniform", 1220 + turn, keys, n, pct)
        if turn == 0 or turn == 3:  # keys that are not there
            rk = O.gen_keys("uniform", 1230 + turn, n)
        if turn == 4:
            ro[rng.random(n) < 0.3] = E.OP_DELETE
        ov, os_ = o.execute_merged(rk, rv, ro, engine=engine)
        gv, gs = g.run(rk, rv, ro)
        assert (gs == os_).all() and (gv == ov).all(), turn
        # and an uncaptured batch between two replays
        rk, rv, ro = O.gen_requests("uniform", 1240 + turn, keys, 100_000, 50)
        ov, os_ = o.execute_merged(rk, rv, ro, engine=engine)
        gv, gs = run_batch(t, rk, rv, ro, mode)
        assert (gs == os_).all() and (gv == ov).all(), turn
    gk, gv = dump(t)
    ok, ovv = o.dump()
    assert (gk == ok).all() and (gv == ovv).all()
    assert (t.leaf_sizes().sum() == gk.size) and t.stats()["error"] == 0


@pytest.mark.parametrize("n", [3_000, 70_000])
def test_empty_build_in_a_graph(gpu, n):
    # a graph that empties the tree and fills it again
    import torch

    t = tree()
    t.bulk_build(dev(np.arange(1, 1000, dtype=np.uint64)), dev(np.arange(1, 1000, dtype=np.uint64)))
    b = empty_u64(n), empty_u64(n), empty_u8(n), empty_u64(n), empty_u8(n)
    none = empty_u64(0)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        s = torch.cuda.current_stream()
        t.bulk_build(none, none, stream=s)
        t.execute(*b, mode=MERGE, stream=s)
    for turn in range(3):
        k, v, op = inserts(1251 + turn, n)
        for x, y in zip(b, (k, v, op)):
            x.copy_(dev(y))
        graph.replay()
        torch.cuda.synchronize()
        assert (host_u8(b[4]) == E.ST_ABSENT).all(), turn
        gk, gv = dump(t)
        o = np.argsort(k)
        assert (gk == k[o]).all() and (gv == v[o]).all(), turn
