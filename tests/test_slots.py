"""The barrier slots of cooperative launches, dealt on the host.

Two launches that may run at the same time must never share a slot: a launch
that stays queued on one stream while thousands pass on others, more streams
than slots, threads, and graphs that give theirs back.
The pool is compiled from the library's own header into a host program.
"""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r'''
#include <cstdio>
#include <set>
#include <thread>
#include "gmes_slots.h"

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
  constexpr int kStreams = 16, kGraphs = 8;
  static volatile uint32_t done[kStreams];
  gmes::SlotPool pool(kStreams, kGraphs, done);
  uint32_t n = 0, queued = 0;
  // a launch waits on stream 7 while 5000 pass on another
  const int held = pool.enter(7, &queued);
  CHECK(held >= 0 && queued == 1);
  for (int k = 0; k < 5000; ++k) {
    const int s = pool.enter(9, &n);
    CHECK(s >= 0 && s != held);
    done[s] = n;  // it has left
  }
  // ... and while many streams come and go
  for (unsigned long long id = 100; id < 3000; ++id) {
    const int s = pool.enter(id, &n);
    CHECK(s >= 0 && s != held);
    done[s] = n;
  }
  CHECK(pool.enter(7, &n) == held && n == 2);  // a stream keeps its slot
  done[held] = 1;                               // the first has left, the second has not
  std::set<int> busy{held};
  for (unsigned long long id = 5000; id < 5000 + kStreams - 1; ++id) {
    const int s = pool.enter(id, &n);
    CHECK(s >= 0 && busy.insert(s).second);
  }
  CHECK(pool.enter(9000, &n) == -1);           // every slot has a launch in flight
  CHECK(pool.enter(7, &n) == held && n == 3);
  done[held] = 3;
  CHECK(pool.enter(9000, &n) == held);          // dealt again once its last has left
  // a slot dealt on: the old stream gets another
  CHECK(pool.enter(7, &n) == -1);
  // graphs: distinct slots beyond the streams', given back and dealt again
  std::set<int> graphs;
  for (int k = 0; k < kGraphs; ++k) {
    const int s = pool.take_graph();
    CHECK(s >= kStreams && s < kStreams + kGraphs && graphs.insert(s).second);
  }
  CHECK(pool.take_graph() == -1);
  pool.give_graph(*graphs.begin());
  CHECK(pool.take_graph() == *graphs.begin());
  // threads, a stream each: nobody ever holds another's slot
  static volatile uint32_t done2[kStreams];
  gmes::SlotPool shared(kStreams, 0, done2);
  volatile int holder[kStreams] = {};
  bool good = true;
  std::thread th[8];
  for (int t = 0; t < 8; ++t)
    th[t] = std::thread([&, t] {
      for (int k = 0; k < 20000; ++k) {
        uint32_t m = 0;
        // every 50 launches a new stream
        const int s = shared.enter(1 + t + 8 * (k / 50), &m);
        if (s < 0 || holder[s] != 0) { good = false; return; }
        holder[s] = t + 1;
        if (holder[s] != t + 1) good = false;
        holder[s] = 0;
        __sync_synchronize();
        done2[s] = m;
      }
    });
  for (auto& x : th) x.join();
  CHECK(good);
  std::printf("ok\n");
  return 0;
}
'''


def test_slots_are_never_shared_in_flight(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    src = tmp_path / "slots.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "slots"
    subprocess.run([cxx, "-std=c++17", "-O2", "-pthread", f"-I{ROOT / 'gmes_gb300' / 'csrc'}",
                    str(src), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout
