"""Waits that the lanes of a warp make one by one, ahead of what a warp does as one (``tcgen05.ld``, ``mma.sync``, ``__syncwarp``): a vote or
a meeting follows, so that all lanes go on together or give up together (CPU, from the sources).  Lanes that leave such a loop by themselves
come together only where the compiler happens to bring them together, and where a wait runs out in some of them, never."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ittai_b200", "csrc")
WAIT = re.compile(r"\b(mbar_try_wait_parked|mbar_try_wait_cluster|mbar_try_wait|mbar_wait_bounded|mbar_wait_abortable|fa_wait)\(")
ONE_LANE = re.compile(r"elect_one\(\)|lane == 0|tid == 0|threadIdx\.x == 0")
MEETING = re.compile(r"__all_sync\(|__syncwarp\(|__syncthreads\(")
WIDE = re.compile(r"\b(tmem_ld_32x\d+|tmem_st_32x\d+|mma16816|ldsm4|ldsm4_t|warp_sum|__any_sync)\(")


def _lonely(text):
    """The waits (their lines) behind which some lanes may go on, or give up, without the others."""
    text = re.sub(r"//[^\n]*", lambda m: " " * len(m[0]), text)
    opened, close, stack = [], {}, []                      # per brace: (open, header)
    for i, ch in enumerate(text):
        if ch == "{":
            stack.append(i)
            opened.append(i)
        elif ch == "}" and stack:
            close[stack.pop()] = i
    header = {i: text[max(text.rfind(c, 0, i) for c in ";{}") + 1:i] for i in opened}
    bad = []
    for m in WAIT.finditer(text):
        around = [i for i in opened if i < m.start() < close.get(i, 0)]
        if re.search(r"__device__[^;{}]*\bbool\s*$", text[:m.start()]) or not around:
            continue                                       # its definition
        if any(ONE_LANE.search(header[i]) for i in around) or any(re.search(r"\bbool\s+\w+\([^)]*\)\s*$", header[i]) for i in around):
            continue                                       # one lane's role, or a helper whose callers are looked at
        statement = text[max(text.rfind(c, 0, m.start()) for c in ";{}") + 1:m.start()]
        if "__all_sync(" in statement:
            continue
        end = text.find(";", m.start())
        brace = text.find("{", m.start(), end)
        leaves = False
        if brace >= 0:                                     # while (!wait) { } is the wait itself; if (!wait) { break; } is its answer
            leaves = "while" not in statement and bool(re.search(r"\b(break|return|continue)\b", text[brace:close[brace]]))
            end = close[brace]
        kernel = [i for i in around if "__global__" in header[i] or "__device__" in header[i]]
        rest = text[end:close[kernel[-1] if kernel else around[0]]]
        meeting, wide = MEETING.search(rest), WIDE.search(rest)
        first = min(x.start() for x in (meeting, wide) if x) if meeting or wide else None
        if first is None:
            continue
        if leaves or wide and wide.start() == first or re.search(r"\b(break|return)\b(?!\s*$)", rest[:first]):
            bad.append(text.count("\n", 0, m.start()) + 1)
    return bad


@pytest.mark.parametrize("source", sorted(os.path.basename(p) for p in glob.glob(os.path.join(CSRC, "*.cu*"))))
def test_lanes_wait_together(source):
    with open(os.path.join(CSRC, source)) as f:
        assert not _lonely(f.read())


def test_the_scan_tells_the_forms_apart():
    kernel = "__global__ void k() { %s }"
    vote = "while (!mbar_try_wait_parked(b, 0)) { if (++n > l) { ok = false; break; } } ok = __all_sync(~0u, ok); if (!ok) break; tmem_ld_32x16(t, v);"
    assert not _lonely(kernel % vote)
    assert _lonely(kernel % vote.replace("ok = __all_sync(~0u, ok);", ""))
    assert not _lonely(kernel % "if (elect_one()) { if (!mbar_wait_bounded(b, 0, l)) { break; } } __syncwarp();")
    assert _lonely(kernel % "for (;;) { if (!mbar_wait_bounded(b, 0, l)) { break; } __syncwarp(); }")
