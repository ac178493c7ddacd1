"""CPU test of the board of solver calls in flight (csrc/rgf_inflight.h)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "rgf_inflight.h"
#include <cassert>
#include <utility>
using rgf::InFlight;
int main() {
  InFlight b;
  int s[4], ev;
  bool over = false;
  auto ask = [&](void* e) { assert(e == &ev); return over; };
  assert(b.others(0, &s[0], 8, ask) == 0);
  {
    InFlight::Ticket a(b, 0, &s[0], 12), c(b, 0, &s[1], 5), other_gpu(b, 1, &s[2], 100);
    assert(b.others(0, &s[0], 8, ask) == 5);          // its own stream's calls follow it
    assert(b.others(0, &s[1], 8, ask) == 12);
    assert(b.others(0, &s[2], 8, ask) == 17);
    assert(b.others(1, &s[3], 8, ask) == 100);
    assert(b.others(0, &s[2], 2, ask) == 12);         // two hardware queues: one call beside this one
    assert(b.others(0, &s[2], 1, ask) == 0);
  }
  assert(b.others(0, &s[2], 8, ask) == 0);            // taken down with the tickets
  InFlight::Ticket kept;
  {
    InFlight::Ticket t(b, 0, &s[0], 7);
    t.until(&ev);
    kept = std::move(t);
  }
  assert(b.others(0, &s[1], 8, ask) == 7);            // outlives its call until the event says so
  over = true;
  assert(b.others(0, &s[1], 8, ask) == 0);
  over = false;
  kept = InFlight::Ticket(b, 0, &s[0], 3);            // replaced by the next call's
  assert(b.others(0, &s[1], 8, ask) == 3);
  kept.reset();
  kept.reset();
  assert(b.others(0, &s[1], 8, ask) == 0);
  return 0;
}
"""


def test_board_counts_the_calls_that_can_run_beside_one(tmp_path):
    src, exe = tmp_path / "board.cpp", tmp_path / "board"
    src.write_text(PROGRAM)
    inc = os.path.join(ROOT, "liteqt_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-pthread", "-I", inc, str(src), "-o", str(exe)],
                   check=True)
    subprocess.run([str(exe)], check=True)
