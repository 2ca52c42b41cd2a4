"""The sweeps' wait for packets (csrc/warp_wait.hpp, the kernel's own code), run by the 32 lanes of a warp against a model of the
warp's vote: also where an earlier wait has run out on some lanes only, every lane casts the same votes and leaves the
wait with the others, and a lane that waits gets what it lacks or the wait ends at its limit on all of them."""
import os
import subprocess

import pytest

from conftest import PKG

MODEL = r"""
#include "warp_wait.hpp"
#include <cstdio>
#include <random>
#include <vector>
// The lanes run one after another, each against the outcomes of the votes that the whole warp would see: a vote is true while
// some lane that waits lacks its packet, which comes after `comes` polls.
int main()
{
    constexpr unsigned limit = 40;
    for (unsigned seed = 0; seed < 20000; seed++) {
        std::mt19937 rng(seed);
        bool ok[32], was[32];
        unsigned comes[32], most = 0;
        for (int l = 0; l < 32; l++) {
            was[l] = ok[l] = rng() % 4 != 0 || seed % 3 == 0;
            comes[l] = rng() % 8 == 0 ? rng() % (2 * limit) : rng() % 6;
            if (ok[l] && comes[l] > most) most = comes[l];
        }
        const unsigned votes = most > limit + 1 ? limit + 2 : most + 1;      // that every lane has to cast
        for (int l = 0; l < 32; l++) {
            unsigned cast = 0, asked = 0;
            gbt::poll_together(ok[l], limit, [&](bool) { return cast++ < most; }, [&] { return asked < comes[l]; }, [&] { asked++; });
            const bool out = most > limit + 1;
            if (cast != votes || ok[l] != (was[l] && !out) || (!was[l] && asked) || (ok[l] && asked < comes[l])) {
                std::printf("seed %u lane %d: %u votes of %u, ok %d, asked %u of %u\n", seed, l, cast, votes, ok[l], asked, comes[l]);
                return 1;
            }
        }
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    d = tmp_path_factory.mktemp("warp")
    (d / "warp.cpp").write_text(MODEL)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(PKG, "csrc"), str(d / "warp.cpp"), "-o", str(d / "warp")], check=True)
    return str(d / "warp")


def test_lanes_vote_alike(model):
    r = subprocess.run([model], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
