"""culda_cgs_b200/csrc/smem_limit.h on the host, with a function in the place of
the CUDA call: a limit is only ever raised, for each kernel and device apart, and
a setting that failed is tried again."""
from __future__ import annotations

import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "culda_cgs_b200" / "csrc"

PROGRAM = r"""
#include "smem_limit.h"
#include <cassert>
#include <thread>
#include <vector>

int main() {
    culda::SmemLimits limits;
    int f = 0, g = 0, calls = 0;
    size_t set[2][2] = {};
    auto raise = [&](int *fn, int device, size_t bytes, int status = 0) {
        return limits.raise(fn, device, bytes, -1, [&](size_t b) {
            ++calls;
            if (status == 0) set[fn == &g][device] = b;
            return status;
        });
    };
    assert(raise(&f, 0, 50000) == 0 && calls == 1 && set[0][0] == 50000);
    assert(raise(&f, 0, 45000) == 0 && calls == 1 && set[0][0] == 50000);  // never lowered
    assert(raise(&f, 0, 50000) == 0 && calls == 1);
    assert(raise(&f, 1, 45000) == 0 && calls == 2 && set[0][1] == 45000);  // another device has its own
    assert(raise(&g, 0, 45000) == 0 && calls == 3 && set[1][0] == 45000);  // and so has another kernel
    assert(raise(&f, 0, 60000, 7) == 7 && calls == 4 && set[0][0] == 50000);
    assert(raise(&f, 0, 60000) == 0 && calls == 5 && set[0][0] == 60000);  // the refused one was not kept

    // what a thread has been granted it keeps, whatever the others ask for
    size_t now = 0;  // written inside the call only
    std::vector<std::thread> team;
    culda::SmemLimits shared;
    for (int t = 0; t < 4; ++t)
        team.emplace_back([&, t] {
            for (int i = 0; i < 20000; ++i) {
                const size_t want = 41000 + 1000 * ((i * 7 + t) % 13);
                assert(shared.raise(&f, 0, want, -1, [&](size_t b) { return assert(b > now), now = b, 0; }) == 0);
            }
        });
    for (std::thread &t : team) t.join();
    assert(now == 53000);
}
"""


def test_limits_are_only_raised(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(CSRC), "-o", str(exe), str(src)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)
