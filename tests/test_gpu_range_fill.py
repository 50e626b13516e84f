"""The two range entries: the filled one zeroes the places past a query's pairs,
the other leaves them as the caller gave them; the pairs and counts are equal."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per", [0, 1, 31, 32, 33, 64, 100, 257])
@pytest.mark.parametrize("n_keys", [0, 1, 5000])
def test_range_fill(gpu, n_keys, per):
    import torch

    rng = np.random.default_rng(per)
    keys = np.arange(1, n_keys + 1).astype(np.uint64) * np.uint64(3)
    t = E.BTree(max_keys=1 << 14, max_batch=1 << 10)
    t.bulk_build(dev(keys), dev(O.value_of(keys)))
    lo = rng.integers(0, 3 * 5000, 333).astype(np.uint64)
    span = rng.integers(0, 3 * max(per, 1) * 2, 333).astype(np.uint64)
    hi = np.where(rng.random(333) < 0.1, np.uint64(0), lo + span)
    lo[0], hi[0] = 0, np.uint64(2**64 - 1)
    got = []
    for name in ("bt_range_batch", "bt_range_batch_filled"):
        k = torch.full((333 * max(per, 1),), -7, dtype=torch.int64, device="cuda")
        v = torch.full_like(k, -7)
        c = torch.full((333,), -7, dtype=torch.int32, device="cuda")
        a, b = dev(lo), dev(hi)
        rc = getattr(E.lib(), name)(t._h, a.data_ptr(), b.data_ptr(), 333, per, k.data_ptr(), v.data_ptr(),
                                    c.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        torch.cuda.synchronize()
        got.append([x.cpu().numpy() for x in (c, k, v)])
    s, e = np.searchsorted(keys, lo), np.searchsorted(keys, hi, side="right")
    want = np.where(lo <= hi, np.maximum(e - s, 0), 0)
    vals = O.value_of(keys)
    for fill, (c, k, v) in enumerate(got):
        assert (c == want).all()
        if per == 0:
            assert (k == -7).all() and (v == -7).all()
            continue
        for i in range(333):
            m = min(int(want[i]), per)
            kk, vv = k[i * per:(i + 1) * per], v[i * per:(i + 1) * per]
            assert (kk[:m].view(np.uint64) == keys[s[i]:s[i] + m]).all()
            assert (vv[:m].view(np.uint64) == vals[s[i]:s[i] + m]).all()
            rest = 0 if fill else -7
            assert (kk[m:] == rest).all() and (vv[m:] == rest).all()
