"""The merge engine's look-back tiles: more of them than there are blocks, their
edges (2048 INSERT keys, 1024 segments), runs of keys of one leaf, old and new
mixed, across the edges; and the gathered writes of the hash front end (16 op
codes a thread) at odd sizes and addresses."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump, run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4096, 148 * 4096, 148 * 4096 + 1, 2 * 148 * 4096 + 77])
def test_inserts_of_many_scan_tiles(gpu, n):
    rng = np.random.default_rng(n)
    base = np.arange(1, 1001, dtype=np.uint64) << np.uint64(52)
    t = E.BTree(max_keys=n + 4096, max_batch=n)
    t.bulk_build(dev(base), dev(base))
    k = rng.permutation(np.arange(n, dtype=np.uint64) * np.uint64(7919) + np.uint64(3))
    v = rng.integers(0, 1 << 62, n).astype(np.uint64)
    run_batch(t, k, v, np.full(n, E.OP_INSERT, np.uint8), E.MODE_SORTED | E.MODE_MERGE_ENGINE)
    gk, gv = dump(t)
    ak, av = np.concatenate([k, base]), np.concatenate([v, base])
    at = np.argsort(ak)
    assert (gk == ak[at]).all() and (gv == av[at]).all()
    assert t.stats()["error"] == 0


@pytest.mark.parametrize("n", [1, 2, 2047, 2048, 2049, 4097, 40_001, 300_000])
@pytest.mark.parametrize("step", [2, 16, 31])
def test_new_keys_among_old_ones_of_their_leaf(gpu, n, step):
    old = np.arange(0, n, step, dtype=np.uint64) + np.uint64(1)
    t = E.BTree(max_keys=2 * n + 4096, max_batch=max(n, 1024))
    t.bulk_build(dev(old), dev(old))
    k = np.random.default_rng(n).permutation(np.arange(n, dtype=np.uint64) + np.uint64(1))
    run_batch(t, k, k + np.uint64(5), np.full(n, E.OP_INSERT, np.uint8), E.MODE_SORTED | E.MODE_MERGE_ENGINE)
    gk, gv = dump(t)
    assert (gk == np.sort(k)).all() and (gv == gk + np.uint64(5)).all()
    assert t.stats()["error"] == 0


@pytest.mark.parametrize("n", [65_537, 65_551, 69_632, 70_001])
@pytest.mark.parametrize("shift", [0, 1, 8])
def test_gathered_writes(gpu, n, shift):
    import torch

    rng = np.random.default_rng(n + shift)
    base = O.gen_keys("uniform", 71, 5_000)
    t = E.BTree(max_keys=1 << 18, max_batch=n)
    o = O.OracleTree()
    t.bulk_build(dev(base), dev(O.value_of(base)))
    o.bulk_build(base, O.value_of(base))
    k = rng.choice(base, n)
    new = rng.random(n) < 0.3
    k[new] = rng.integers(1, 1 << 62, int(new.sum())).astype(np.uint64)
    v = rng.integers(0, 1 << 62, n).astype(np.uint64)
    op = rng.choice([E.OP_INSERT, E.OP_GET, E.OP_DELETE], n, p=[0.05, 0.9, 0.05]).astype(np.uint8)
    ov, os_ = o.execute_merged(k, v, op, engine=O.ENGINE_MERGE)
    ops = torch.zeros(n + 16, dtype=torch.uint8, device="cuda")[shift:shift + n]
    ops.copy_(dev(op))
    gv, gs = torch.empty_like(dev(v)), torch.empty_like(ops)
    t.execute(dev(k), dev(v), ops, gv, gs, mode=E.MODE_SORTED | E.MODE_MERGE_ENGINE)
    assert (gs.cpu().numpy() == os_).all()
    assert (gv.cpu().numpy().view(np.uint64) == ov).all()
