"""The calls that enumerate the leaves, on trees of no leaf, one leaf and two."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 2, 24, 25, 48])  # 24 keys to a leaf
def test_few_leaves(gpu, n):
    keys = np.sort(O.gen_keys("uniform", 1601, 48))[:n]
    t = E.BTree(max_keys=1 << 10, max_batch=64)
    for _ in range(2):  # the second turn on a new tree in the same rows
        t.bulk_build(dev(keys), dev(O.value_of(keys)))
        leaves = -(-n // 24)
        assert t.leaf_sizes().tolist() == [n // leaves + (i < n % leaves) for i in range(leaves)]
        assert t.level_counts().tolist() == ([] if n == 0 else [1] if leaves == 1 else [leaves, 1])
        assert t.stats(with_leaves=True)["n_leaves"] == leaves
        gk, gv = dump(t)
        assert (gk == keys).all() and (gv == O.value_of(keys)).all()


def test_counts_then_builds(gpu):
    # nothing of a count is left running in the build's memory
    keys = np.sort(O.gen_keys("uniform", 1611, 3_000))
    t = E.BTree(max_keys=1 << 14, max_batch=4_096)
    for n in (1, 3_000, 20, 2_999, 24, 25) * 20:
        t.bulk_build(dev(keys[:n]), dev(O.value_of(keys[:n])))
        assert t.level_counts()[0] == -(-n // 24) and t.size() == n
    gk, gv = dump(t)
    assert (gk == keys[:25]).all() and (gv == O.value_of(keys[:25])).all()
