"""Sizes of the small batches' clusters: a device that takes smaller clusters than
sixteen blocks runs smaller batches in them and the rest on the general path."""
import ctypes

import pytest

import eirene_b200 as E

PER_BLOCK = 4096


@pytest.fixture(scope="module")
def rules():
    lib = E.lib()
    cluster, limit = lib._ZN2bt13small_clusterEmj, lib._ZN2bt11small_limitEj
    cluster.argtypes, cluster.restype = [ctypes.c_size_t, ctypes.c_uint], ctypes.c_uint
    limit.argtypes, limit.restype = [ctypes.c_uint], ctypes.c_size_t
    return cluster, limit


def test_sixteen_blocks_as_measured(rules):
    cluster, limit = rules
    assert limit(16) == 65_536
    assert [cluster(n, 16) for n in (1, 128, 129, 256, 257, 1024, 1025, 65_536)] == [1, 1, 2, 2, 4, 8, 16, 16]


@pytest.mark.parametrize("most", [0, 1, 2, 4, 8, 16])
def test_no_block_gets_more_than_it_holds(rules, most):
    cluster, limit = rules
    for n in {1, 2, 127, 128, 129, 1000, 1024, 1025, limit(most) - 1, limit(most)}:
        if 1 <= n <= limit(most):
            c = cluster(n, most)
            assert 1 <= c <= most and c & (c - 1) == 0 and c * PER_BLOCK >= n
    assert limit(0) == 0  # no cluster at all: every batch is too large


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1_000, 65_536])
def test_this_device_takes_sixteen_blocks(gpu, n):
    # three kernels are the small batches' form
    import torch

    from tests.helpers import empty_u8, empty_u64

    t = E.BTree(max_keys=1 << 18, max_batch=1 << 16)
    k, op, out = empty_u64(n), empty_u8(n), (empty_u64(n), empty_u8(n))
    before = E.launch_count()
    t.execute(k, k, op, *out, mode=E.MODE_SORTED | E.MODE_MERGE_ENGINE)
    torch.cuda.synchronize()
    assert E.launch_count() - before == 3
