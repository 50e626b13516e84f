"""Calls of one handle on different streams, where the first one is documented
to be synchronous: the second one meets what the first one left."""
import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.helpers import dev, empty_u64, empty_u8, host_u8

pytestmark = pytest.mark.gpu


def busy(stream, cycles=200_000_000):
    """About a tenth of a second of work ahead of the next call on `stream`."""
    import torch

    with torch.cuda.stream(stream):
        torch.cuda._sleep(cycles)


@pytest.mark.parametrize("n", [100, 100_000])  # both plain lookup forms
def test_empty_build_is_done_when_it_returns(gpu, n):
    import torch

    keys = O.gen_keys("uniform", 1101, n)
    t = E.BTree(max_keys=1 << 18, max_batch=1 << 17)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    q, none = dev(keys), empty_u64(0)
    ov, os_ = empty_u64(n), empty_u8(n)
    torch.cuda.synchronize()
    for _ in range(2):  # the first turn loads the kernels, which waits for the device
        t.bulk_build(q, dev(O.value_of(keys)))
        t.search(q, ov, os_, stream=s2)
        torch.cuda.synchronize()
        assert (host_u8(os_) == E.ST_FOUND).all()
        busy(s1)
        t.bulk_build(none, none, stream=s1)
        t.search(q, ov, os_, stream=s2)
        s2.synchronize()
        assert (host_u8(os_) == E.ST_ABSENT).all()
    assert t.size() == 0


@pytest.mark.parametrize("call", ["range", "search", "execute"])
def test_loaded_image_is_whole_when_it_returns(gpu, tmp_path, call):
    # the separators' prefixes and the leaves' fingerprints, which the file does
    # not hold: a lookup on one stream must not be the one that makes them for
    # a call on another
    import torch

    n = 100_000
    keys = np.sort(O.gen_keys("uniform", 1111, n))
    a = E.BTree(max_keys=1 << 18, max_batch=1 << 17)
    a.bulk_build(dev(keys), dev(O.value_of(keys)))
    path = str(tmp_path / "tree.img")
    a.save_image(path)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    q = dev(keys)
    ov, os_ = empty_u64(n), empty_u8(n)
    get = torch.full((n,), E.OP_GET, dtype=torch.uint8, device="cuda")

    def check(t):
        if call == "range":
            counts, k, _ = t.range(q[:1000], q[3:1003], 4, stream=s2)
            s2.synchronize()
            assert (counts == 4).all() and (k[:, 0] == q[:1000]).all()
            return
        os_.fill_(9)
        torch.cuda.current_stream().synchronize()
        if call == "search":
            t.search(q, ov, os_, stream=s2)
        else:
            t.execute(q, q, get, ov, os_, mode=E.MODE_SORTED | E.MODE_MERGE_ENGINE, stream=s2)
        s2.synchronize()
        assert (host_u8(os_) == E.ST_FOUND).all()

    check(a)
    for _ in range(2):  # the first turn loads the kernels, which waits for the device
        b = E.BTree(max_keys=1 << 18, max_batch=1 << 17)
        b.load_image(path)
        o1, st1 = empty_u64(n), empty_u8(n)
        torch.cuda.synchronize()
        busy(s1)
        b.search(q, o1, st1, stream=s1)
        check(b)
        torch.cuda.synchronize()
        assert (host_u8(st1) == E.ST_FOUND).all()


@pytest.mark.parametrize("n, max_batch", [(1_000, 1_024), (70_000, 1 << 17)])
def test_new_handle_beside_a_busy_default_stream(gpu, n, max_batch):
    # everything that a new handle, its first dump and its first training clear is
    # clear when they are used, whatever else the default stream holds
    import torch

    keys = np.sort(O.gen_keys("uniform", 1121, n))
    k, v, op = dev(keys), dev(O.value_of(keys)), torch.full((n,), E.OP_INSERT, dtype=torch.uint8, device="cuda")
    s = torch.cuda.Stream()
    ov, os_ = empty_u64(n), empty_u8(n)
    for _ in range(2):  # the first turn loads the kernels, which waits for the device
        torch.cuda.synchronize()
        busy(torch.cuda.default_stream())
        t = E.BTree(max_keys=1 << 18, max_batch=max_batch)
        t.execute(k, v, op, ov, os_, mode=E.MODE_SORTED | E.MODE_MERGE_ENGINE, stream=s)
        t.sync(s)
        t.retrain(stream=s)
        s.synchronize()
        assert (host_u8(os_) == E.ST_ABSENT).all()
        gk, gv = t.dump()
        assert (gk == k).all() and (gv == v).all()
        t.close()
