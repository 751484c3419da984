"""The cache of free page-locked blocks, compiled by itself: blocks of two
devices side by side, a replaced context, the limit."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dygrass_b200", "csrc")

PROGRAM = r"""
#include "pinned_cache.h"
#include <cstdio>
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
    static char m[16];
    // handles on two devices closed in turn: no block of the other is lost
    dyg::PinnedCache c(100);
    CHECK(c.keep(0, 11, m + 0, 10));
    CHECK(c.keep(1, 22, m + 1, 10));
    CHECK(c.keep(0, 11, m + 2, 20));
    CHECK(c.keep(1, 22, m + 3, 20));
    CHECK(c.total() == 60);
    CHECK(c.take(0, 11, 10) == m + 0 && c.take(1, 22, 10) == m + 1);
    CHECK(c.take(0, 11, 20) == m + 2 && c.take(1, 22, 20) == m + 3);
    CHECK(c.total() == 0);
    // neither another device's block, nor another size, nor a dead context's
    CHECK(c.keep(0, 11, m + 4, 10));
    CHECK(!c.take(1, 11, 10) && !c.take(0, 11, 11) && !c.take(0, 12, 10));
    // device 0 was reset: its old blocks are forgotten, device 1's stay
    CHECK(c.keep(1, 22, m + 5, 10));
    CHECK(c.keep(0, 12, m + 6, 10));
    CHECK(c.total() == 20);
    CHECK(c.take(0, 12, 10) == m + 6 && c.take(1, 22, 10) == m + 5);
    // the limit
    CHECK(c.keep(0, 12, m + 7, 100) && !c.keep(0, 12, m + 8, 1) && c.total() == 100);
    return 0;
}
"""


def test_pinned_cache(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    cp = subprocess.run([gxx, "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", CSRC, str(src), "-o", str(exe)],
                        capture_output=True, text=True)
    assert cp.returncode == 0, cp.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
