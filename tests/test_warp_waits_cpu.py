"""The warm-start network's waits on barriers: a wait that a whole warp acts on is decided for the warp (mbar_wait_warp), as what
follows it, a load of tensor memory, needs all lanes on one path; only the waits of one elected lane are not."""
import os
import re

from conftest import PKG


def _span(text, at):
    """the braces' block that opens at or after `at`"""
    depth, first = 0, text.index("{", at)
    for n in range(first, len(text)):
        depth += {"{": 1, "}": -1}.get(text[n], 0)
        if depth == 0:
            return first, n
    raise AssertionError("unbalanced braces")


def test_waits_of_a_warp_are_voted():
    text = open(os.path.join(PKG, "csrc", "warmstart.cu")).read()
    alone = [_span(text, m.start()) for m in re.finditer(r"if \(lane == 0[^\n]*\) \{\n|bool mbar_wait_warp\(", text)]
    calls = [m.start() for m in re.finditer(r"(?<!bool )\bmbar_wait_bounded\(", text)]
    assert len(calls) >= 10
    stray = [text.count("\n", 0, c) + 1 for c in calls if not any(a < c < b for a, b in alone)]
    assert not stray, f"lines {stray}"
