"""The solves' status words: device code changes them by atomic operations only (kernels of two streams set bits of one
word side by side)."""
import glob
import os
import re

from conftest import PKG


def test_status_words_are_changed_atomically():
    plain = []
    for f in sorted(glob.glob(os.path.join(PKG, "csrc", "*.cu")) + glob.glob(os.path.join(PKG, "csrc", "*.cuh"))):
        for n, line in enumerate(open(f), 1):
            if re.search(r"(\bB\.st\[[^]]*\]|\bst)\.status\s*(\||&|\^)?=", line):
                plain.append(f"{os.path.basename(f)}:{n}")
    assert not plain
