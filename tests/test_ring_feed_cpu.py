"""The order in which the sweeps' input ring asks for its copies (csrc/ring_feed.hpp, the kernel's own code), run against a
model of the stages' barriers: copies that land at once, late or after every wait has run out, consumers that give
up waiting (and then say no more that they are done with a step). No barrier may be armed twice in a phase, no copy may start over one that has not
landed, and every copy that lands before the waits of the drain run out has landed when the drain returns."""
import os
import subprocess

import pytest

from conftest import PKG

MODEL = r"""
#include "ring_feed.hpp"
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
constexpr int kStages = 3, kGroup = 2, kLimit = 100;
struct Bar { int phase = 0, group = -1; long lands = -1; };       // lands: time of the armed phase's copies
int main(int argc, char **argv)
{
    const int steps = std::atoi(argv[1]), slow = std::atoi(argv[2]), lost = std::atoi(argv[3]);
    for (unsigned seed = 0; seed < 2000; seed++) {
        std::mt19937 rng(seed);
        auto pick = [&](int n) { return (int)(rng() % (unsigned)n); };
        Bar bar[kStages];
        long now = 0;
        auto settle = [&] {
            for (auto &b : bar)
                if (b.group >= 0 && now >= b.lands) { b.phase++; b.group = -1; }
        };
        bool ok = true, waits = true;
        auto wait_on = [&](int s, unsigned parity, bool &good) {
            for (int q = 0; good && q < kLimit; q++, now++) {
                settle();
                if ((unsigned)(bar[s].phase & 1) != parity) return;
            }
            good = false;
        };
        gbt::RingFeed<kStages> feed{(steps + kGroup - 1) / kGroup};
        bool fault = false;
        auto ask = [&](int g, int s) {
            settle();
            if (bar[s].group >= 0 || g != bar[s].phase * kStages + s) fault = true;
            bar[s].group = g;
            bar[s].lands = now + (slow && pick(6) == 0 ? pick(4 * kLimit) : pick(5));
        };
        for (int s = 0; s < kStages; s++) feed.next(ok, ask);
        for (int n = 0; n < steps && !fault; n++) {
            // the consumers wait for the step's inputs; they give up where these do not land, or another tile's
            // terms do not come
            wait_on(n / kGroup % kStages, (unsigned)(n / kGroup / kStages) & 1u, waits);
            if (lost && pick(30) == 0) waits = false;
            now += pick(3);
            // the feeding thread waits for their word, which does not come then, or comes too late
            if (!waits) { now += kLimit; ok = false; }
            if (slow && pick(40) == 0) ok = false;
            if ((n + 1) % kGroup == 0) feed.next(ok, ask);
        }
        bool last = true;
        feed.drain([&](int s, unsigned parity) { wait_on(s, parity, last); });
        bool flying = false;
        for (auto &b : bar) flying = flying || b.group >= 0;
        if (fault || (last && flying) || (!slow && !lost && (!ok || feed.asked != feed.groups))) {
            std::printf("seed %u: fault %d, flying %d, drained %d, asked %d of %d\n", seed, fault, flying, last, feed.asked, feed.groups);
            return 1;
        }
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    src, exe = d / "ring.cpp", d / "ring"
    src.write_text(MODEL)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(PKG, "csrc"), str(src), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("steps", [1, 2, 5, 6, 7, 13, 64, 141])
@pytest.mark.parametrize("slow", [0, 1])
@pytest.mark.parametrize("lost", [0, 1])
def test_copies_in_order(model, steps, slow, lost):
    r = subprocess.run([model, str(steps), str(slow), str(lost)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
