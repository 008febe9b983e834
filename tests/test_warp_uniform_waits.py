"""CPU test: a wait that may give up never splits a warp of the network kernels.

A bounded wait (role_wait) can end differently for the lanes of a warp: one sees the phase complete,
another the abort flag or its own time limit.  What follows a reader's wait is .sync.aligned (ldmatrix,
mma.sync, tcgen05.ld) or a warp barrier, so the whole warp has to take one decision; a single-thread
role may decide alone.  Read off the source: the path itself runs only when a copy never arrives.
"""

import os
import re

SRC = os.path.join(os.path.dirname(__file__), "..", "fast-light-field_gb300", "csrc", "flf_net.cu")


def blocks_at(text, pos):
    """Headers of the braces that enclose text[pos], outermost first."""
    stack, start = [], 0
    for i, ch in enumerate(text[:pos]):
        if ch == "{":
            stack.append(text[start:i])
            start = i + 1
        elif ch == "}":
            if stack:
                stack.pop()
            start = i + 1
        elif ch == ";" and text[start:i].count("(") == text[start:i].count(")"):
            start = i + 1
    return stack


def statement_at(text, pos):
    a = max(text.rfind(c, 0, pos) for c in ";{}")
    return text[a + 1:text.index(";", pos)]


def source():
    with open(SRC) as f:
        t = re.sub(r"//[^\n]*", "", f.read())
    return re.sub(r'"(?:[^"\\]|\\.)*"', '""', t)


def test_waits_of_whole_warps_take_one_decision():
    text = source()
    calls = [m.start() for m in re.finditer(r"\brole_wait\(", text)]
    assert len(calls) >= 12
    for pos in calls:
        around = blocks_at(text, pos)
        stmt = statement_at(text, pos)
        if "bool role_wait(" in text[pos - 5:pos + 10] or any("lane == 0" in h for h in around):
            continue
        if "__all_sync(0xffffffffu" in stmt:
            continue
        var = re.search(r"(\w+) = (?:\1 && )?role_wait", stmt)
        assert var and re.search(r"__all_sync\(0xffffffffu, %s\b" % var.group(1), text[pos:pos + 1000]), stmt


def test_abort_flag_is_read_by_the_warp_as_one():
    """A loop that a whole warp leaves on the abort flag reads it once for the warp."""
    text = source()
    for m in re.finditer(r"\bfor \(([^;{}]*);([^;{}]*\*abort_s[^;{}]*);", text):
        if any("lane == 0" in h for h in blocks_at(text, m.start())):
            continue
        cond = m.group(2)
        assert "__any_sync(0xffffffffu, *abort_s)" in cond, cond
