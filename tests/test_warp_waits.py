"""Bounded waits in the tcgen05 kernels, read from their sources: where a whole warp waits, its lanes go on alike.  A wait that runs out may run out
for some lanes of a warp only (one sees the abort flag, another its barrier), and lanes that part there never meet again at the aligned
instructions behind it (tensor-memory loads, barriers, shuffles): the bound of the wait would be none."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpt_fast_b200", "csrc")


def waits(text):
    """(line, name, by one lane) of every call of mbar_wait or mbar_wait_warp outside of the helpers themselves.  A call is one lane's where
    a block around it, or the statement that it belongs to, begins with a test of the lane."""
    text = re.sub(r"//[^\n]*", lambda m: " " * len(m.group()), text)
    found, blocks, start = [], [], 0                     # blocks: the text in front of every open brace
    calls = {m.start(): m.group(1) for m in re.finditer(r"\b(mbar_wait(?:_warp)?)\(", text)}
    for i, ch in enumerate(text):
        if ch == "{":
            blocks.append(text[start:i])
            start = i + 1
        elif ch == "}":
            blocks.pop()
            start = i + 1
        elif ch == ";":
            start = i + 1
        if i in calls and blocks:                        # (at file level: the helpers' own heads)
            around = blocks + [text[start:i]]
            if not any(re.search(r"bool (?:mbar_wait|$)", b) for b in around):
                one = any(re.search(r"\blane == 0\b|\bthreadIdx\.x == 0\b|\btid == 0\b", b) for b in around)
                found.append((text.count("\n", 0, i) + 1, calls[i], one))
    return found


def test_it_sees_both_kinds():
    code = """__device__ bool mbar_wait(int b) { return mbar_wait(b); }
    void k() { if (warp == 0) { if (lane == 0) { auto f = [&]() { return mbar_wait(1); }; } } else { for (;;) { ok = mbar_wait(2); mbar_wait_warp(3); } } }"""
    assert waits(code) == [(2, "mbar_wait", True), (2, "mbar_wait", False), (2, "mbar_wait_warp", False)]


@pytest.mark.parametrize("source", ["attention_tc.cu", "gemm_split.cu", "gemm_tc.cu"])
def test_whole_warps_wait_alike(source):
    found = waits(open(os.path.join(CSRC, source)).read())
    assert len(found) >= 7
    wrong = [(line, name) for line, name, one in found if one == (name == "mbar_wait_warp")]
    assert not wrong, f"{source}: {wrong}"


def test_no_other_source_waits_on_barriers_of_its_own():
    others = [f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and f not in ("attention_tc.cu", "gemm_split.cu", "gemm_tc.cu")]
    assert not [f for f in others if re.search(r"\bmbar_wait\(", open(os.path.join(CSRC, f)).read())]
