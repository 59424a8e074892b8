"""A bounded wait may run out in one lane of a warp and not in the next.  Code that
a whole warp runs must therefore wait through mbar_wait_warp, whose result is one
for all lanes; mbar_wait_bounded is left to roles of a single thread.  Read from
the kernels' sources: running a wait out in the middle of a kernel is no test."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ca3dmm_b200", "csrc")
# headers of blocks that one thread alone enters
SINGLE = re.compile(r"if \((threadIdx\.x == 0|lane == 0|producer)\b[^|]*\)\s*$|auto issue_one = \[&\]\(\) -> bool\s*$")


def sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and f != "k_common.cuh")


def plain(text):
    return re.sub(r'//[^\n]*|"(\\.|[^"\\])*"', "", text)


def enclosing(text, pos):
    """Headers of the blocks around pos, and the statement that pos stands in."""
    stack, start = [], 0
    for i, c in enumerate(text[:pos]):
        if c == "{":
            stack.append(text[start:i].strip())
        elif c == "}":
            stack.pop()
        if c in "{};":
            start = i + 1
    return stack + [text[start:pos].strip()]


@pytest.mark.parametrize("name", sources())
def test_single_lane_waits_stay_in_single_thread_roles(name):
    text = plain(open(os.path.join(CSRC, name)).read())
    for m in re.finditer(r"\bmbar_wait_bounded\(", text):
        around = enclosing(text, m.start())
        # the wait itself may be the last operand of such a condition
        single = any(SINGLE.search(h) for h in around[:-1]) or re.search(
            r"if \((threadIdx\.x == 0|lane == 0|producer) &&\s*!?$", around[-1])
        assert single, (name, around)


def test_refills_run_in_the_producer_thread():
    """The refill lambda holds a single-thread wait: every call of it does, too."""
    text = plain(open(os.path.join(CSRC, "k_dgemm.cu")).read())
    calls = [m.start() for m in re.finditer(r"\bissue_one\(\)", text)]
    assert len(calls) == 3
    for pos in calls:
        around = enclosing(text, pos)
        assert any(re.search(r"if \(producer\)", h) for h in around), around
