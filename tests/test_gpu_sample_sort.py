"""The sample sort of the touched requests (BT_OPT_TOUCH_SORT 1) against the
oracle at the edges of its buckets (1024 pairs per bucket, waves of 148, 512
buckets, 4096 pairs in a block), and against the radix sort (0) where buckets
outgrow a block; hot keys, one key only, ascending and descending requests,
reserved keys and invalid op codes."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, dump, run_batch

pytestmark = pytest.mark.gpu
MERGE = E.MODE_SORTED | E.MODE_MERGE_ENGINE


def make(rng, n, law):
    if law == "ascending":
        rk = np.sort(rng.integers(0, 1 << 63, n).astype(np.uint64))
    elif law == "descending":
        rk = np.sort(rng.integers(0, 1 << 63, n).astype(np.uint64))[::-1].copy()
    elif law == "one":
        rk = np.full(n, 12345, np.uint64)
    elif law == "hot":
        rk = rng.integers(0, 1 << 63, n).astype(np.uint64)
        hot = rng.integers(0, 1 << 63, 5).astype(np.uint64)
        at = rng.random(n) < 0.7
        rk[at] = hot[rng.integers(0, 5, int(at.sum()))]
    elif law == "near":  # keys that share their high 40 bits, many of them repeated
        rk = np.uint64(0x77 << 40) + rng.integers(0, n, n).astype(np.uint64)
    else:
        rk = rng.integers(0, 1 << 63, n).astype(np.uint64)
    ro = rng.choice([E.OP_INSERT, E.OP_GET, E.OP_DELETE, 5], n, p=[0.7, 0.15, 0.14, 0.01]).astype(np.uint8)
    rk[rng.random(n) < 0.002] = E.KEY_MAX
    return rk, rng.integers(0, 1 << 62, n).astype(np.uint64), ro


@pytest.mark.parametrize("law", ["uniform", "ascending", "descending", "one", "hot", "near"])
@pytest.mark.parametrize("n", [1, 1023, 1025, 1500, 2049, 70_000, 200_000, 270_000])
def test_sample_sort_matches_oracle(gpu, n, law):
    rng = np.random.default_rng(n)
    keys = O.gen_keys("uniform", 71, 20_000)
    t = E.BTree(max_keys=1 << 20, max_batch=max(n, 1024))
    t.set_option(E.OPT_TOUCH_SORT, 1)
    o = O.OracleTree()
    t.bulk_build(dev(keys), dev(O.value_of(keys)))
    o.bulk_build(keys, O.value_of(keys))
    for b in range(2):
        rk, rv, ro = make(rng, n, law)
        ov, os_ = o.execute_merged(rk, rv, ro, engine=O.ENGINE_MERGE)
        gv, gs = run_batch(t, rk, rv, ro, MERGE)
        assert (gs == os_).all() and (gv == ov).all(), b
    gk, gvv = dump(t)
    ok, ovv = o.dump()
    assert (gk == ok).all() and (gvv == ovv).all()
    assert t.stats()["error"] == 0


@pytest.mark.parametrize("law", ["uniform", "hot", "near", "descending"])
@pytest.mark.parametrize("n", [524_289, 700_001, 1 << 21, 3_000_000])
def test_sample_sort_beyond_its_buckets_matches_radix(gpu, n, law):
    import torch

    out = []
    for opt in (1, 0):
        rng = np.random.default_rng(n)
        t = E.BTree(max_keys=n + (1 << 18), max_batch=n)
        t.set_option(E.OPT_TOUCH_SORT, opt)
        rk, rv, ro = make(rng, n, law)
        k, v, o = dev(rk), dev(rv), dev(ro)
        ov, os_ = torch.empty_like(k), torch.empty_like(o)
        t.execute(k, v, o, ov, os_, mode=MERGE)
        out.append((ov.cpu(), os_.cpu(), *(x.cpu() for x in t.dump())))
        assert t.stats()["error"] == 0
        t.close()
    for a, b in zip(*out):
        assert torch.equal(a, b)
