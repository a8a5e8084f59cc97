"""A push block's counters (kpt_tally.h), host build: the words carry, and the
judge's evaluations stay the count of served substeps when a block gives up
with particles in flight."""
from __future__ import annotations

import os
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "kokkos-particletransport_gb300", "csrc")
SOURCE = """
#include "kpt_tally.h"
#include <cstdio>
#define CHECK(c) if (!(c)) { std::puts(#c); return 1; }
int main() {
    using namespace kpt;
    BlockTally b{};
    unsigned long long served = 0, fallbacks = 0, steps = 0;
    // particles of 0 .. 39 substeps, every third substep a fallback; the block
    // gives up on the last ten, some of which only ever fell back
    for (int particle = 0; particle < 40; ++particle) {
        const bool abandoned = particle >= 30, only_fallbacks = particle >= 35;
        for (int k = 0; k < particle; ++k) {
            const bool out = only_fallbacks || k % 3 == 0;
            if (out) tally_add(b.fallbacks, 1u);
            (out ? fallbacks : served) += 1;
        }
        if (abandoned) {
            tally_abandon(b, particle);
        } else {
            tally_finish(b, particle, particle == 7 ? 2 : 0);
        }
        steps += particle;
        CHECK(tally_evaluations(b) == served);
    }
    CHECK(tally_word(b.steps) == steps && tally_word(b.fallbacks) == fallbacks);
    CHECK(b.pushed == 40 && b.failed == 1 && b.max_steps == 29);
    // a block that gives up at once, with nothing finished
    BlockTally none{};
    for (int k = 0; k < 5; ++k) tally_add(none.fallbacks, 1u);
    tally_abandon(none, 5);
    CHECK(tally_evaluations(none) == 0 && none.pushed == 1 && none.max_steps == 0);
    // the low words carry
    BlockTally big{};
    for (int k = 0; k < 3; ++k) tally_finish(big, 0x7fffffff, 0);
    tally_add(big.fallbacks, 0xffffffffu);
    tally_add(big.fallbacks, 2u);
    CHECK(tally_word(big.steps) == 3ull * 0x7fffffffull);
    CHECK(tally_word(big.fallbacks) == 0x100000001ull);
    CHECK(tally_evaluations(big) == 3ull * 0x7fffffffull - 0x100000001ull);
    return 0;
}
"""


def test_counters(tmp_path):
    src, exe = tmp_path / "tally.cpp", tmp_path / "tally"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", CSRC, str(src), "-o",
                    str(exe)], check=True)
    done = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert done.returncode == 0, done.stdout
