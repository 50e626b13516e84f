"""The merge engine's scans when the live entries need more tiles (4096) than
there are blocks: one batch of INSERTs into a small tree, read back whole."""
import numpy as np
import pytest

import eirene_b200 as E
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
