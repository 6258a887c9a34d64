"""Kernels that are launched chained may start before the kernel ahead of them
has finished: what that kernel wrote may only be read after chainWait(), and
nothing may tell the compiler that it never changes."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "fullc0ntact_gb300", "csrc")
# kernel -> the loads through the read-only path that it may make, of data that no
# kernel ahead of it writes: the training samples (its first launch of a call is
# not chained)
READ_ONLY = {"kSdfTrain": {"samples + idx", "shapes + idx", "&samples[idx].w"}}


def _close(text, i, pair):
    depth = 0
    for k in range(i, len(text)):
        depth += (text[k] == pair[0]) - (text[k] == pair[1])
        if depth == 0:
            return k
    raise AssertionError("unbalanced")


def _chained():
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"__global__\s+void\s+(__launch_bounds__)?", text):
            i = m.end()
            if m.group(1):
                i = _close(text, text.index("(", i), "()") + 1
            name = re.match(r"\s*(\w+)\s*", text[i:])
            p0 = text.index("(", i)
            p1 = _close(text, p0, "()")
            b0 = text.index("{", p1)
            body = text[b0:_close(text, b0, "{}") + 1]
            if "chainWait()" in body:
                out.append((name.group(1), text[p0:p1 + 1], body))
    return out


def test_chained_kernels_are_found():
    names = {n for n, _, _ in _chained()}
    assert {"kIntegrate", "kScanCellsOwn", "kFixupGather", "kCollideRows", "kSdfReduce",
            "kIntegrateDistMap"} <= names


@pytest.mark.parametrize("kernel", _chained(), ids=lambda k: k[0])
def test_no_pointer_is_promised_to_be_unaliased(kernel):
    assert "__restrict__" not in kernel[1]


@pytest.mark.parametrize("kernel", _chained(), ids=lambda k: k[0])
def test_no_read_only_loads(kernel):
    name, _, body = kernel
    loads = set(re.findall(r"(?:__ldg|ldg4)\(([^()]*)\)", body))
    assert loads <= READ_ONLY.get(name, set())


@pytest.mark.parametrize("kernel", _chained(), ids=lambda k: k[0])
def test_trigger_and_wait_come_before_shared_data(kernel):
    """chainTrigger() then chainWait(), once each, before any early return, store
    or atomic."""
    name, _, body = kernel
    assert body.count("chainTrigger()") == 1 and body.count("chainWait()") == 1
    assert body.index("chainTrigger()") < body.index("chainWait()")
    assert not re.search(r"\breturn\s*;|atomic\w+\(", body[:body.index("chainWait()")])
