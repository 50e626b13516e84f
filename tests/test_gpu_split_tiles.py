"""Batches parted in two lists by tiles of 1024 requests: the tile's edges, tiles
that are all one class, and odd remainders, for the hash front end against the
oracle and for STM batches (distinct keys) against a dictionary."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump, run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("write", [0.0, 0.05, 1.0])
@pytest.mark.parametrize("n", [65_537, 66_559, 66_560, 66_561])
def test_front_tiles_match_oracle(gpu, n, write):
    rng = np.random.default_rng(n)
    base = O.gen_keys("uniform", 71, 10_000)
    t = E.BTree(max_keys=1 << 18, max_batch=n)
    o = O.OracleTree()
    t.bulk_build(dev(base), dev(O.value_of(base)))
    o.bulk_build(base, O.value_of(base))
    k, v = rng.choice(base, n), rng.integers(0, 1 << 62, n).astype(np.uint64)
    op = np.where(rng.random(n) < write, rng.choice([E.OP_INSERT, E.OP_DELETE], n), E.OP_GET).astype(np.uint8)
    op[: n // 3] = E.OP_GET  # whole tiles of lookups
    ov, os_ = o.execute_merged(k, v, op, engine=O.ENGINE_MERGE)
    gv, gs = run_batch(t, k, v, op, E.MODE_SORTED | E.MODE_MERGE_ENGINE)
    assert (gs == os_).all() and (gv == ov).all()


@pytest.mark.parametrize("write", [0.0, 0.1, 1.0])
@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 5_121])
def test_stm_tiles_match_dictionary(gpu, n, write):
    rng = np.random.default_rng(n)
    pool = np.unique(rng.integers(0, 1 << 63, 3 * n + 64).astype(np.uint64))
    rng.shuffle(pool)
    base = pool[: n // 2 + 8]
    t = E.BTree(max_keys=1 << 16, max_batch=max(n, 1024))
    t.bulk_build(dev(base), dev(O.value_of(base)))
    d = dict(zip(base.tolist(), O.value_of(base).tolist()))
    k = rng.permutation(np.concatenate([base[: n // 2], pool[base.size:]])[:n])
    v = rng.integers(0, 1 << 62, n).astype(np.uint64)
    op = np.where(rng.random(n) < write, E.OP_INSERT, E.OP_GET).astype(np.uint8)
    gv, gs = run_batch(t, k, v, op, E.MODE_STM)
    for i, (kk, vv, oo) in enumerate(zip(k.tolist(), v.tolist(), op.tolist())):
        assert (gs[i], gv[i]) == ((E.ST_FOUND, d[kk]) if kk in d else (E.ST_ABSENT, 0)), i
        if oo == E.OP_INSERT:
            d[kk] = vv
    assert dump(t)[0].tolist() == sorted(d)
