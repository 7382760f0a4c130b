"""Buffers allocated as a group (csrc/alloc_group.h): whichever allocation fails, none is kept and
no pointer stays set, and the next attempt succeeds.  Host code alone, against a fake allocator."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "alloc_group.h"
static int live = 0, calls = 0, fail_at = -1;
static bool get(void** p, size_t b) {
  if (calls++ == fail_at) { *p = (void*)1; return false; }   // (a failed call may leave anything there)
  *p = std::malloc(b); ++live; return true;
}
static void put(void* p) { std::free(p); --live; }
int main() {
  for (int f = 0; f < 4; ++f) {
    void *a = nullptr, *b = nullptr, *c = nullptr, *d = nullptr;
    calls = 0; fail_at = f;
    const bool ok = cfd::alloc_group({{&a, 8}, {&b, 16}, {&c, 24}, {&d, 32}}, get, put);
    std::printf("%d %d %d\n", ok, (a != nullptr) + (b != nullptr) + (c != nullptr) + (d != nullptr), live);
    fail_at = -1;
    const bool again = cfd::alloc_group({{&a, 8}, {&b, 16}, {&c, 24}, {&d, 32}}, get, put);
    std::printf("%d %d %d\n", again, (a != nullptr) + (b != nullptr) + (c != nullptr) + (d != nullptr), live);
    for (void* p : {a, b, c, d}) put(p);
  }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_all_or_none(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "cfd3d_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")[:-1]
    assert out == ["0 0 0", "1 4 4"] * 4
