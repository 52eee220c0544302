"""The side-stream copy of host targets (rmesh_b200/csrc/side_copy.h) against a fake
runtime whose calls fail one at a time: a failed set-up leaves nothing behind and is
started again, and a copy that may be under way is waited for before the memory is
anyone else's."""
from __future__ import annotations

import os
import subprocess

from conftest import ROOT

SRC = r'''
#include "side_copy.h"
#include <cstdio>
#include <cstdlib>
#include <set>
#include <vector>
static int fail_at = -1, calls = 0, next_id = 1, copying = 0, waits = 0;
static std::set<int> streams, events;
static int step() { return calls++ == fail_at ? 7 : 0; }
struct Fake {
  using Error = int;
  using Stream = int;
  using Event = int;
  static int create_stream(int* s) { if (step()) return 7; streams.insert(*s = next_id++); return 0; }
  static int create_event(int* e) { if (step()) return 7; events.insert(*e = next_id++); return 0; }
  static int record(int e, int) { if (!events.count(e)) abort(); return step(); }
  static int wait(int, int e) { if (!events.count(e)) abort(); return step(); }
  static int copy(void*, const void*, size_t, int s) { if (!streams.count(s)) abort(); if (step()) return 7; copying = 1; return 0; }
  static void synchronize(int s) { if (!streams.count(s)) abort(); ++waits; copying = 0; }
  static void destroy_event(int e) { if (!events.erase(e)) abort(); }
  static void destroy_stream(int s) { if (!streams.erase(s)) abort(); }
};
#define CHECK(x) do { if (!(x)) { printf("line %d, call %d fails: %s\n", __LINE__, fail_at, #x); return 1; } } while (0)
int main() {
  // 3 calls set up, 2 order the copy behind the main stream, 3 copy
  for (fail_at = -1; fail_at < 8; ++fail_at) {
    calls = copying = waits = 0;
    {
      rm::SideCopy<Fake> c;
      int e = c.open();
      CHECK((e != 0) == (fail_at >= 0 && fail_at < 3));
      if (e) {
        CHECK(streams.empty() && events.empty());
        CHECK(c.open() == 0);  // started again, whole
      }
      CHECK(streams.size() == 1 && events.size() == 2);
      CHECK(c.open() == 0 && streams.size() == 1);  // once
      e = c.follow(100);
      if (!e) e = c.copy(nullptr, nullptr, 1, 100);
      CHECK((e != 0) == (fail_at >= 3));
      if (e) {  // the caller's exit on an error
        c.settle();
        CHECK(!copying && !c.in_flight());
        CHECK(fail_at < 6 || waits == 1);
        CHECK(c.follow(100) == 0 && c.copy(nullptr, nullptr, 1, 100) == 0);
      }
      CHECK(c.in_flight());
      if (fail_at % 2) c.landed();  // the main stream was waited for
    }
    CHECK(streams.empty() && events.empty());
    CHECK(fail_at % 2 || !copying);  // the end waits for a copy that nobody waited for
  }
  puts("ok");
}
'''


def test_every_call_may_fail(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(SRC)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "rmesh_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.stdout.strip() == "ok", out.stdout
