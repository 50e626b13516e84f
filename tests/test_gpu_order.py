"""Calls of one handle on different streams, where the first one is documented
to be synchronous: the second one meets what the first one left."""
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
