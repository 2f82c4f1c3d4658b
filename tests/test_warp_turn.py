"""The decision of a persistent warp that holds one system per lane
(csrc/warp_turn.h), compiled for the host and driven through every way a batch
can begin and end: the work list runs out, systems arrive finished, the time
slice ends at any turn, the first one included.  The warp has to end, may not
step while nothing is active, and writes every claimed system back once."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "coupled-bubble-control_b200", "csrc")

HARNESS = r"""
#include <stdio.h>
#include <stdlib.h>
#include "warp_turn.h"
// One warp over `n` systems, system s taking len[s] steps (0: finished when
// loaded); lanes past `slots` take none; from turn `deadline` on (< 0: never)
// every system stops and none is claimed.  0: ends as it should.
static int warp(int n, const int* len, int slots, int deadline) {
  int sys[32], left[32], head = 0;
  int written[256] = {0}, claimed[256] = {0};
  bool drained[32];
  for (int l = 0; l < 32; ++l) sys[l] = -1, left[l] = 0, drained[l] = l >= slots;
  for (int turn = 0; turn < 100000; ++turn) {
    unsigned active = 0, held = 0, done = 0;
    for (int l = 0; l < 32; ++l) {
      if (deadline >= 0 && turn >= deadline) drained[l] = true, left[l] = 0;
      active |= (unsigned)(sys[l] >= 0 && left[l] > 0) << l;
      held |= (unsigned)(sys[l] >= 0) << l;
      done |= (unsigned)drained[l] << l;
    }
    switch (cbc::next_turn(active, held, done)) {
      case cbc::Turn::exit:
        for (int s = 0; s < n; ++s)
          if (claimed[s] != written[s] || claimed[s] > 1 || (deadline < 0 && !claimed[s])) return 1;
        return 0;
      case cbc::Turn::refill:
        for (int l = 0; l < 32; ++l) {
          if (sys[l] >= 0 && left[l] == 0) ++written[sys[l]], sys[l] = -1;
          if (sys[l] >= 0 || drained[l]) continue;
          if (head < n) ++claimed[head], left[l] = len[head], sys[l] = head++;
          else drained[l] = true;
        }
        break;
      case cbc::Turn::step:
        if (!active) return 2;
        for (int l = 0; l < 32; ++l) if (active >> l & 1) --left[l];
    }
  }
  return 3;
}
int main() {
  srand(1);
  for (int it = 0; it < 20000; ++it) {
    const int n = rand() % 100, slots = it % 3 ? 32 : 1 + rand() % 32, deadline = it % 4 ? rand() % 40 : -1;
    int len[100];
    for (int s = 0; s < n; ++s) len[s] = rand() % 5 ? 1 + rand() % 30 : 0;
    for (int k = 0; k < 2; ++k) {
      const int d = k ? 0 : deadline;
      const int e = warp(n, len, slots, d);
      if (e) { printf("n %d slots %d deadline %d: error %d\n", n, slots, d, e); return 1; }
    }
  }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_warp_ends_from_every_start(tmp_path):
    src, exe = tmp_path / "turn.cpp", tmp_path / "turn"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


def test_lane_per_system_worker_steps_only_after_that_decision():
    """The exit is taken before the refill block, so no block can skip it."""
    text = open(os.path.join(CSRC, "ensemble_kernel.cuh")).read()
    body = text[text.index("ensemble_solo_kernel("):text.index("ensemble_duo_kernel(")]
    body = re.sub(r"//[^\n]*", "", body)
    at = [body.index(x) for x in ("next_turn(", "Turn::exit) break;", "Turn::refill) {", "solo_step(")]
    assert at == sorted(at)
    assert body.count("break;") == 1
