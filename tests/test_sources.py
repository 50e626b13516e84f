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


def functions():
    """(file, name, signature, body) of the device functions and kernels."""
    for f, text in sources():
        for m in re.finditer(r"\b__(?:global|device)__\b", text):
            end = text.find("{", m.start())
            if end < 0 or ";" in text[m.start():end] or text[m.start():end].lstrip("_ ").startswith("__global__ __device__"):
                continue
            sig = text[m.start():end]
            name = re.findall(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\s*\([^)]*\)", "", sig))
            if not name:
                continue
            depth, i = 1, end + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield f, name[0], sig, text[end:i]


def test_dependent_launches_read_nothing_early():
    # a kernel that is resident before the one in front of it has ended, and
    # whatever it calls, makes ordinary loads: a __restrict__ pointer lets the
    # compiler move a load ahead of the wait, and ld.global.nc reads a path that
    # the wait says nothing about
    by_name = {}
    for f, name, sig, body in functions():
        by_name.setdefault(name, []).append((f, sig, body))
    todo = [n for n, d in by_name.items()
            if any("__global__" in s and re.search(r"\b(after_previous|wait_for_previous)\s*\(", b) for _, s, b in d)]
    assert len(todo) > 20  # the parser still finds them
    seen, bad = set(), []
    while todo:
        n = todo.pop()
        if n in seen:
            continue
        seen.add(n)
        for f, sig, body in by_name[n]:
            if "__restrict__" in sig or re.search(r"\b__ldg\s*\(|ld\.global\.nc", body):
                bad.append(f"{f}: {n}")
            todo += [w for w in set(re.findall(r"\b(\w+)\s*(?:<[^;{}()]*>)?\s*\(", body)) if w in by_name]
    assert not bad, sorted(bad)
