"""The host's look at the rows that a kernel is about to read (csrc/host_rows.hpp): it ends, on the host, at any page of
the range that is not mapped or not readable, also one between its ends, and touches nothing outside it."""
import os
import signal
import subprocess

import pytest

from conftest import PKG

PROGRAM = r"""
#include "host_rows.hpp"
#include <cstdio>
#include <cstdlib>
#include <sys/mman.h>
// pages of a mapping, the one to close (-1: none; how: 0 unmapped, 1 not readable), first byte and length of the range
int main(int argc, char **argv)
{
    const long page = sysconf(_SC_PAGESIZE), pages = std::atol(argv[1]), hole = std::atol(argv[2]);
    char *m = (char *)mmap(nullptr, (size_t)(pages * page), PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (m == MAP_FAILED) return 2;
    if (hole >= 0 && (std::atoi(argv[3]) ? mprotect(m + hole * page, (size_t)page, PROT_NONE) : munmap(m + hole * page, (size_t)page))) return 2;
    gbt::read_every_page(m + std::atol(argv[4]), (size_t)(std::atol(argv[5]) + std::atol(argv[6]) * page));
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("rows")
    (d / "rows.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(PKG, "csrc"), str(d / "rows.cpp"), "-o", str(d / "rows")], check=True)
    return str(d / "rows")


def _run(program, *a):
    return subprocess.run([program] + [str(x) for x in a]).returncode


@pytest.mark.parametrize("how", [0, 1])
@pytest.mark.parametrize("hole", [0, 1, 5, 8, 9])
@pytest.mark.parametrize("first", [0, 4, 36])
def test_ends_at_a_hole(program, how, hole, first):
    assert _run(program, 10, hole, how, first, 64, 9) == -signal.SIGSEGV


@pytest.mark.parametrize("args", [(10, -1, 0, 0, 0, 10),        # the whole mapping
                                  (10, 9, 1, 8, -8, 9),         # up to the last byte before a closed page
                                  (10, 9, 0, 0, 0, 9),
                                  (10, 1, 1, 100, 28, 0),       # within a page
                                  (10, 0, 1, 0, 0, 0)])         # nothing
def test_reads_nothing_outside(program, args):
    assert _run(program, *args) == 0
