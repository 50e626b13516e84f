"""Device memory that bulk builds of more than max_batch keys keep: one share for
all handles of a device, given back with the last of them; builds of several
handles at a time, from several threads and streams."""
import subprocess
import sys
import threading

import numpy as np
import pytest

import eirene_b200 as E
from oracle import oracle as O
from tests.conftest import ROOT
from tests.helpers import dev, dump, host_u64

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def free_mib():
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()  # not what the tests' own tensors leave cached
    return torch.cuda.mem_get_info()[0] / MIB


def handle():
    return E.BTree(max_keys=1 << 22, max_batch=1_024)


def test_scratch_is_shared_and_given_back(gpu):
    # in a process of its own: another test's handle may still hold the device's scratch
    r = subprocess.run([sys.executable, "-c", "import tests.test_gpu_build_scratch as t; t.shared_and_given_back()"],
                       capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


def shared_and_given_back():
    n = 3_000_001  # about 110 MiB of scratch
    keys = O.gen_keys("uniform", 1501, n)
    k, v = dev(keys), dev(O.value_of(keys))
    handle().close()  # what the first handle of a process leaves
    start = free_mib()
    trees = [handle() for _ in range(4)]
    made = free_mib()
    kept = []
    for t in trees:
        before = free_mib()
        t.bulk_build(k, v)
        kept.append(before - free_mib())
    assert kept[0] > 50, kept
    assert max(kept[1:]) < 8, kept
    assert made - free_mib() < 1024 + 8
    # the ones that are left still build when others go
    for t in trees[:3]:
        t.close()
        trees[3].bulk_build(k, v)
    order = np.argsort(keys)
    gk, gv = dump(trees[3])
    assert (gk == keys[order]).all() and (gv == O.value_of(keys)[order]).all()
    del gk, gv
    trees[3].close()
    assert start - free_mib() < 8


def test_builds_of_several_threads(gpu):
    import torch

    sizes = [2_000, 700_001, 1_500_000, 3_000_001]
    data = [O.gen_keys("uniform", 1511 + i, n) for i, n in enumerate(sizes)]
    dd = [(dev(k), dev(O.value_of(k))) for k in data]
    torch.cuda.synchronize()
    errors = []

    def work(i):
        try:
            s = torch.cuda.Stream()
            for turn in range(6):
                t = handle()
                k, v = dd[(i + turn) % len(dd)]
                t.bulk_build(k, v, stream=s)
                assert t.size() == k.numel()
                if turn % 3 == 0:
                    gk, gv = t.dump()
                    keys = data[(i + turn) % len(data)]
                    order = np.argsort(keys)
                    assert (host_u64(gk) == keys[order]).all() and (host_u64(gv) == O.value_of(keys)[order]).all()
                t.close()
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
