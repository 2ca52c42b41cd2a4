"""The solves' status words: every bit that a kernel may set is described in the public header, and device code changes
the words by atomic operations only (kernels of two streams set bits of one word side by side)."""
import glob
import os
import re

from conftest import PKG, ROOT


def test_header_describes_every_bit():
    common = open(os.path.join(PKG, "csrc", "gbt_common.cuh")).read()
    bits = re.findall(r"GBT_STATUS_\w+ = (\d+)", common)
    assert len(bits) == 4
    header = open(os.path.join(ROOT, "include", "gbturbo.h")).read()
    text = re.search(r"/\*((?:(?!\*/).)*?)\*/\s*int gb_get_status", header, re.S).group(1)
    missing = [b for b in bits if not re.search(rf"\bbit {b}\b", text)]
    assert not missing


def test_status_words_are_changed_atomically():
    plain = []
    for f in sorted(glob.glob(os.path.join(PKG, "csrc", "*.cu")) + glob.glob(os.path.join(PKG, "csrc", "*.cuh"))):
        for n, line in enumerate(open(f), 1):
            if re.search(r"(\bB\.st\[[^]]*\]|\bst)\.status\s*(\||&|\^)?=", line):
                plain.append(f"{os.path.basename(f)}:{n}")
    assert not plain
