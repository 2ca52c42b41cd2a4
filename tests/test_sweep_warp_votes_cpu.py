"""The sweeps' incoming warp polls for packets by a vote of its 32 lanes: a lane's wait on a barrier that runs out there must have
run out on all of them, or some lanes would vote where others do not. So that warp waits by bar_wait_warp only, and what
leaves its poll loop is the warp's outcome too."""
import os
import re

from conftest import PKG


def _block(text, head):
    first = text.index(head)
    depth, at = 0, text.index("{", first)
    for n in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[n], 0)
        if depth == 0:
            return text[at:n]
    raise AssertionError("unbalanced braces")


def test_incoming_warp_waits_together():
    text = open(os.path.join(PKG, "csrc", "wavefront.cu")).read()
    incoming = _block(text, "} else if (warp == 4) {")
    assert "__any_sync(0xffffffffu, late)" in incoming
    assert re.findall(r"\bbar_wait\w*", incoming) == ["bar_wait_warp"]
    loop = _block(incoming, "for (unsigned polls = 0; ok; polls++) {")
    assert re.findall(r"if \(([^;]*)\) (?:break|\{ ok = false; break; \});", loop) == ["!__any_sync(0xffffffffu, late)"]
    assert "if (polls > kWaitLimit) { ok = false; break; }" in loop
    helper = _block(text, "void bar_wait_warp(unsigned bar, unsigned parity, bool &ok)")
    assert re.search(r"bar_wait\(bar, parity, ok\);\s*ok = __all_sync\(0xffffffffu, ok\)", helper)
