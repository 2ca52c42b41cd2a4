"""Work split over host threads (csrc/host_threads.hpp) where starting one fails: every part is done all the same, each
once, and the process goes on."""
import os
import subprocess

import pytest

from conftest import PKG

PROGRAM = r"""
#include "host_threads.hpp"
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
struct Few {
    int *left;
    template <typename F> std::thread operator()(F f) const
    {
        if ((*left)-- == 0) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
        return std::thread(std::move(f));
    }
};
int main(int, char **argv)
{
    const size_t n = (size_t)std::atoi(argv[1]);
    int left = std::atoi(argv[2]);
    std::vector<std::atomic<int>> done(n);
    gbt::in_parallel(n, [&](size_t t) { done[t]++; }, Few{&left});
    for (auto &d : done) if (d != 1) return 1;
    // an exception of the caller's own part leaves after the threads are joined
    std::atomic<int> others{0};
    left = std::atoi(argv[2]);
    try {
        gbt::in_parallel(n, [&](size_t t) { if (t == 0) throw std::runtime_error("part 0"); others++; }, Few{&left});
        return n == 0 ? 0 : 2;
    } catch (const std::runtime_error &) {
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("threads")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(PKG, "csrc"), str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("parts", [0, 1, 2, 7, 16])
@pytest.mark.parametrize("started", [0, 1, 3, 100])
def test_every_part_is_done(program, parts, started):
    assert subprocess.run([program, str(parts), str(started)], timeout=60).returncode == 0
