"""The bounded waits of the triangular solves (csrc/warp_wait.h), run on the host:
32 lanes as threads that need not run in step and see a value at different
polls.  Whatever they see, all lanes have to come to the same collectives in the
same order, and a value that never comes has to end the wait."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "cfdsfemmpi_b200" / "csrc"

PROGRAM = r"""
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <random>
#include <thread>
#include <vector>
#include "warp_wait.h"

constexpr int LANES = 32;

// A full-mask collective: every lane has to arrive, and at the same place.
struct Warp {
  std::mutex mu;
  std::condition_variable cv;
  int site = 0, in = 0, any = 0, all = 1, r_any = 0, r_all = 1;
  unsigned long gen = 0;
  bool wrong = false;
  bool vote(int where, bool v, bool want_any)
  {
    std::unique_lock<std::mutex> lk(mu);
    if (in == 0) { site = where; any = 0; all = 1; }
    if (site != where) wrong = true;
    any |= v; all &= v;
    if (++in == LANES) {
      in = 0; r_any = any; r_all = all; gen++;
      cv.notify_all();
    } else {
      const unsigned long g = gen;
      if (!cv.wait_for(lk, std::chrono::seconds(10), [&] { return gen != g || wrong; })) wrong = true;
    }
    if (wrong) { cv.notify_all(); std::printf("lanes at different collectives (%d, %d)\n", site, where); std::fflush(stdout); std::_Exit(1); }
    return want_any ? r_any : r_all;
  }
};

struct Shared {
  std::atomic<int> gave_up{0}, gives{0};
  std::atomic<unsigned long long> clock{0};
};
struct Env {
  Shared *s;
  unsigned long long step;
  bool gave_up() const { return s->gave_up != 0; }
  void give_up() const { s->gave_up = 1; s->gives++; }
  unsigned long long now() const { return s->clock += step; }
};

// mode 0: values come; 1: the value polled for never comes; 2: one of a row's other values never comes
bool round(unsigned seed, int mode)
{
  Warp w;
  Shared sh;
  std::vector<std::thread> t;
  std::atomic<int> left{0}, got{0};
  for (int lane = 0; lane < LANES; lane++)
    t.emplace_back([&, lane] {
      std::mt19937 g(seed * 97 + lane);
      // polls after which this lane sees the value: around the times when the waits look at the clock
      const int seen = mode == 1 ? 1 << 30 : 1 + (int)(g() % 3 ? g() % 2500 : 1020 + g() % 8);
      const int whole = mode == 2 && lane == 7 ? 1 << 30 : (int)(g() % 100);
      cfdgpu::LaneWait<Env> wait{{&sh, mode ? 2000000000ull : 1ull}};
      int polls = 0, tries = 0;
      cfdgpu::wait_lanes([&] { return ++polls >= seen; }, wait, [&] { w.vote(1, true, true); });
      cfdgpu::retry_warp([&] { return w.vote(2, ++tries <= whole, true); }, wait,
                         [&](bool v) { return w.vote(3, v, false); });
      w.vote(4, true, true);
      if (polls >= seen && tries > whole) got++;
      left++;
    });
  for (auto &x : t) x.join();
  if (left != LANES) return false;
  if (mode == 0) return got == LANES && sh.gives == 0;
  return sh.gave_up == 1 && sh.gives >= 1;
}

int main()
{
  for (int mode = 0; mode < 3; mode++)
    for (unsigned seed = 0; seed < (mode == 2 ? 1u : 8u); seed++)
      if (!round(seed, mode)) { std::printf("mode %d seed %u: wrong outcome\n", mode, seed); return 1; }
  std::printf("ok\n");
  return 0;
}
"""


def test_lanes_leave_a_wait_together_and_a_wait_ends(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    src, exe = tmp_path / "wait.cpp", tmp_path / "wait"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", str(CSRC), "-o", str(exe), str(src)], check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.strip() == "ok", p.stdout + p.stderr
