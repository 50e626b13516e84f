"""Bulk build and enumeration with their counts on the device: shapes, contents
and errors against the oracle, at the sizes where a level starts to need a
launch of its own (512 nodes), with the handle's work buffers (n <= max_batch)
and with its pool, repeated keys, and fills down to one child per node."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump, empty_u64

pytestmark = pytest.mark.gpu


def check(t, o):
    gk, gv = dump(t)
    ok, ov = o.dump()
    assert gk.size == ok.size and (gk == ok).all() and (gv == ov).all()
    assert (t.leaf_sizes() == o.leaf_sizes()).all()
    assert (t.level_counts() == o.level_counts()).all()
    assert t.stats(True)["n_leaves"] == o.leaf_sizes().size


@pytest.mark.parametrize("max_batch", [1024, 1 << 20])
@pytest.mark.parametrize("leaf_fill, inner_fill, n", [
    (24, 24, 1), (24, 24, 24), (24, 24, 25), (24, 24, 1024), (24, 24, 1025), (24, 24, 24 * 512), (24, 24, 24 * 512 + 1),
    (24, 24, 24 * 25 * 512), (24, 24, 24 * 25 * 512 + 1), (31, 31, 700_000), (2, 1, 3), (2, 1, 5000), (3, 2, 20_000)])
def test_build_shapes(gpu, leaf_fill, inner_fill, n, max_batch):
    rng = np.random.default_rng(n)
    keys = np.unique(rng.integers(0, 1 << 63, n + n // 50 + 8).astype(np.uint64))[:n]
    rng.shuffle(keys)
    t = E.BTree(max_keys=8 * n + 8192, max_batch=max_batch, leaf_fill=leaf_fill, inner_fill=inner_fill)
    o = O.OracleTree(leaf_fill, inner_fill)
    for dup in (False, True, False):
        k = keys
        if dup:  # half of the keys twice, the last value wins
            k = np.concatenate([keys[: n // 2], keys, keys[: n // 3]])
        v = rng.integers(0, 1 << 62, k.size).astype(np.uint64)
        t.bulk_build(dev(k), dev(v))
        o.bulk_build(k, v)
        check(t, o)


@pytest.mark.parametrize("max_batch", [1024, 1 << 17])
def test_build_errors_leave_an_empty_tree(gpu, max_batch):
    t = E.BTree(max_keys=1 << 16, max_batch=max_batch)
    keys = np.arange(1, 50_001).astype(np.uint64)
    vals = O.value_of(keys)
    for bad, code in ((np.append(keys, np.uint64(E.KEY_MAX)), -5), (np.arange(1, 3_000_001).astype(np.uint64), -4)):
        t.bulk_build(dev(keys), dev(vals))
        assert t.size() == keys.size
        with pytest.raises(E.BTError) as e:
            t.bulk_build(dev(bad), dev(bad))
        assert e.value.code == code
        assert t.size() == 0 and t.level_counts().size == 0
    t.bulk_build(dev(keys), dev(vals))
    gk, gv = dump(t)
    assert (gk == keys).all() and (gv == vals).all()


def test_dump_into_too_small_a_buffer(gpu):
    import ctypes

    t = E.BTree(max_keys=1 << 16, max_batch=1 << 14)
    keys = np.arange(1, 10_001).astype(np.uint64)
    t.bulk_build(dev(keys), dev(keys))
    k, v = empty_u64(9_999), empty_u64(9_999)
    n = ctypes.c_size_t(0)
    rc = E.lib().bt_dump_sorted(t._h, k.data_ptr(), v.data_ptr(), 9_999, ctypes.byref(n), None)
    assert rc == -4 and n.value == 10_000
    assert int(k.abs().sum()) == 0 and int(v.abs().sum()) == 0
