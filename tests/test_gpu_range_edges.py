"""Range scans whose ends lie on the borders of leaves and of their parents,
in trees of one leaf, two levels and more, with keys that share their high 32
bits (full separators instead of prefixes), after inserts and deletes."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump, run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 40])
@pytest.mark.parametrize("n", [1, 24, 25, 600, 601, 24 * 25 * 25 + 1])
def test_range_borders(gpu, n, shift):
    import torch

    keys = (np.arange(1, n + 1).astype(np.uint64) * np.uint64(4)) << np.uint64(shift)
    t = E.BTree(max_keys=1 << 17, max_batch=1 << 12)
    t.bulk_build(dev(keys), dev(O.value_of(keys)))
    for step in range(2):
        gk, gv = dump(t)
        edge = np.concatenate([[0], np.cumsum(t.leaf_sizes())])[:-1].astype(np.int64)
        edge = np.unique(np.clip(np.concatenate([edge, edge - 1, edge + 1, edge[::25], [gk.size - 1]]), 0, gk.size - 1))
        a = edge[np.random.default_rng(n).permutation(edge.size)[:400]]
        lo = np.repeat(gk[a], 4)
        hi = np.concatenate([np.array([gk[x], gk[min(x + 23, gk.size - 1)], gk[min(x + 700, gk.size - 1)], gk[x] + np.uint64(1)])
                             for x in a])
        lo = np.concatenate([lo, lo - np.uint64(1), lo + np.uint64(1)])
        hi = np.concatenate([hi, hi - np.uint64(1), hi])
        for per in (0, 1, 40, 800):
            c, k, v = t.range(dev(lo), dev(hi), per)
            torch.cuda.synchronize()
            s, e = np.searchsorted(gk, lo), np.searchsorted(gk, hi, side="right")
            want = np.where(lo <= hi, np.maximum(e - s, 0), 0)
            assert (c.cpu().numpy() == want).all()
            k, v = k.cpu().numpy().view(np.uint64), v.cpu().numpy().view(np.uint64)
            for i in range(0, lo.size, 7):
                m = min(int(want[i]), per)
                assert (k[i, :m] == gk[s[i]:s[i] + m]).all() and (v[i, :m] == gv[s[i]:s[i] + m]).all()
                assert not k[i, m:].any() and not v[i, m:].any()
        # emptied leaves and split ones
        gone = keys[(keys.size // 3):(keys.size // 3) + 60]
        more = (np.arange(1, 200).astype(np.uint64) * np.uint64(4) + np.uint64(1)) << np.uint64(shift)
        rk = np.concatenate([gone, more])
        ro = np.concatenate([np.full(gone.size, E.OP_DELETE), np.zeros(more.size)]).astype(np.uint8)
        run_batch(t, rk, O.value_of(rk), ro, E.MODE_SORTED | E.MODE_MERGE_ENGINE)
