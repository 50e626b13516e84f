"""Rules of the CUDA sources that no run on a quiet GPU would show broken."""
import os
import re

from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "eirene_b200", "csrc")


def sources():
    for f in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, f)).read()
        # without comments, every line kept
        text = re.sub(r"/\*.*?\*/", lambda m: "\n" * m.group().count("\n"), text, flags=re.S)
        yield f, re.sub(r"//[^\n]*", "", text)


def test_nothing_is_cleared_on_the_default_stream():
    # cudaMemset of device memory is queued on the default stream and returns: the
    # handle's streams and its callers' do not wait for it
    found = [f"{f}:{text[:m.start()].count(chr(10)) + 1}" for f, text in sources()
             for m in re.finditer(r"\bcudaMemset\s*\(", text)]
    assert not found, found
