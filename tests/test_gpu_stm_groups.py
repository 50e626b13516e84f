"""STM writes four to a warp (group_write): batches without repeated keys, so
that the answers and the contents follow from a dictionary, at the edges of a
warp's window and with many requests per leaf (lock conflicts, full and emptied
leaves), with GETs, deletes of absent keys and invalid requests among them."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump, run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("combine", [1, 0])
@pytest.mark.parametrize("tree", [0, 20, 3000])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 32, 33, 900, 20_000])
def test_stm_writes_match_dictionary(gpu, n, tree, combine):
    rng = np.random.default_rng(n + tree)
    pool = np.unique(rng.integers(0, 1 << 63, 2 * n + tree + 64).astype(np.uint64))
    rng.shuffle(pool)
    keys = pool[:tree]
    t = E.BTree(max_keys=1 << 18, max_batch=1 << 15)
    t.set_option(E.OPT_STM_COMBINE, combine)
    if tree:
        t.bulk_build(dev(keys), dev(O.value_of(keys)))
    d = dict(zip(keys.tolist(), O.value_of(keys).tolist()))
    for b in range(4):
        have = np.array(list(d), np.uint64)
        rk = np.unique(np.concatenate([have[rng.integers(0, have.size, n)] if have.size else pool[:0],
                                       pool[rng.integers(0, pool.size, n)]]))
        rng.shuffle(rk)
        rk = rk[:n]
        rv = rng.integers(0, 1 << 62, rk.size).astype(np.uint64)
        ro = rng.choice([E.OP_INSERT, E.OP_DELETE, E.OP_GET, 9], rk.size, p=[0.6, 0.25, 0.1, 0.05] if b % 2 else
                        [0.2, 0.6, 0.15, 0.05]).astype(np.uint8)
        if rk.size > 2:
            rk[1] = E.KEY_MAX
        gv, gs = run_batch(t, rk, rv, ro, E.MODE_STM)
        for i, (k, v, o) in enumerate(zip(rk.tolist(), rv.tolist(), ro.tolist())):
            if o > 2 or k == E.KEY_MAX:
                assert gs[i] == E.ST_REJECTED
                continue
            assert (gs[i], gv[i]) == ((E.ST_FOUND, d[k]) if k in d else (E.ST_ABSENT, 0)), (b, i, o)
            if o == E.OP_INSERT:
                d[k] = v
            elif o == E.OP_DELETE:
                d.pop(k, None)
        gk, gvv = dump(t)
        assert gk.tolist() == sorted(d) and gvv.tolist() == [d[k] for k in sorted(d)]
        assert t.size() == len(d) and t.stats()["error"] == 0
