"""One lock per CUDA context (csrc/ctx_slots.h): a thread that uses one context's slot holds up
another user of the same context and nobody else.  Host code alone."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "ctx_slots.h"
int main() {
  cfd::CtxSlots<int> m;
  std::printf("%d\n", m.find(1) == nullptr);
  auto* a = m.put(1, 10);
  auto* b = m.put(2, 20);
  std::printf("%d %d\n", a->value, b->value);
  // a slot that another thread made first is kept
  std::printf("%d %d\n", m.put(1, 99) == a, a->value);
  std::lock_guard<std::mutex> hold(a->mu);
  std::atomic<int> got{0}, same{-1};
  std::thread t([&] {
    { std::lock_guard<std::mutex> l(m.find(2)->mu); got = 1; }   // (would wait for ever on one lock for all)
    { std::lock_guard<std::mutex> l(m.put(3, 30)->mu); got = 2; }
    same = m.find(1)->mu.try_lock();
  });
  t.join();
  std::printf("%d %d\n", got.load(), same.load());
  std::vector<std::thread> ts;
  std::atomic<int> bad{0};
  for (int q = 0; q < 8; ++q)
    ts.emplace_back([&] {
      for (unsigned long long c = 10; c < 200; ++c) {
        auto* s = m.find(c);
        if (!s) s = m.put(c, (int)c);
        if (s->value != (int)c || m.find(c) != s) ++bad;
      }
    });
  for (auto& x : ts) x.join();
  std::printf("%d\n", bad.load());
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_contexts_do_not_wait_for_one_another(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-pthread", "-I", os.path.join(ROOT, "cfd3d_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.split("\n")[:-1]
    assert out == ["1", "10 20", "1 10", "2 0", "0"]
