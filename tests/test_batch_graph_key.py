"""The key under which a batch keeps its captured interval loop (kpt_rules.h),
on the host: everything the captured launches hold by value is in it."""
from __future__ import annotations

import os
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "kokkos-particletransport_gb300", "csrc")
SOURCE = """
#include "kpt_rules.h"
#include <cstdio>
#define CHECK(c) if (!(c)) { std::puts(#c); return 1; }
int main() {
    using namespace kpt;
    char memory[8];
    const BatchGraphShape shape{3, 16, 0, 1, 128, 1, false};
    const std::vector<BatchGraphRun> runs = {{100, memory, memory + 1, memory + 2},
                                             {50, memory + 3, memory + 4, memory + 5}};
    const auto key = batch_graph_key(shape, runs);
    CHECK(key == batch_graph_key(shape, runs));
    for (size_t r = 0; r < runs.size(); ++r) {
        auto grown = runs;       // an injection, a split, an upload
        grown[r].count += 1;
        CHECK(key != batch_graph_key(shape, grown));
        for (int k = 0; k < 3; ++k) {  // a buffer that was freed and taken anew
            auto moved = runs;
            (k == 0 ? moved[r].order : k == 1 ? moved[r].keys : moved[r].tile_counts) = memory + 7;
            CHECK(key != batch_graph_key(shape, moved));
        }
    }
    auto fewer = runs;
    fewer.pop_back();
    CHECK(key != batch_graph_key(shape, fewer));
    const BatchGraphShape other[] = {{4, 16, 0, 1, 128, 1, false}, {3, 8, 0, 1, 128, 1, false},
                                     {3, 16, 3, 1, 128, 1, false}, {3, 16, 0, 2, 128, 1, false},
                                     {3, 16, 0, 1, 64, 1, false},  {3, 16, 0, 1, 128, 2, false},
                                     {3, 16, 0, 1, 128, 1, true}};
    for (const BatchGraphShape& s : other) CHECK(key != batch_graph_key(s, runs));
    return 0;
}
"""


def test_key_holds_counts_and_buffers(tmp_path):
    src, exe = tmp_path / "key.cpp", tmp_path / "key"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", CSRC, str(src), "-o",
                    str(exe)], check=True)
    done = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert done.returncode == 0, done.stdout
