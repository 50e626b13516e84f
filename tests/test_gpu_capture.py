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
