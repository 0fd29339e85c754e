"""The slots a sweep's compute warp stages its chunks in (sweep_ahead, sc_sweep.cuh), on
the CPU: copies in flight to one place are not ordered, so no slot may get a copy before
its last one has landed, and a chunk must find its own data.  The warp's walk over its
tiles is played with the kernel's own rule for what is copied ahead, for both stage
depths, all short tiles and some long ones, tiles that are not swept, and the next
ticket known early, late or not at all.  The same walk with a zero fill in place of a
copy that is left out must be caught."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_SRC = r'''
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "sc_sweep.cuh"
struct Slot { long chunk = -1; long commit = -1; bool read = true; };
// 0: sound; 1: a copy into a slot with a copy in flight; 2: unread data overwritten; 3: wrong data read
int play(int D, int NC, unsigned seed, bool fill) {
  const int DG = D / 4, NG = (NC + 3) / 4;
  std::srand(seed);
  std::vector<Slot> slot(D);
  long commits = 0, landed = 0;  // groups of copies committed; those with a smaller number have landed
  auto write = [&](int s, long chunk) {
    if (slot[s].commit >= landed) return 1;
    if (!slot[s].read) return 2;
    slot[s] = {chunk, commits, chunk < 0};
    return 0;
  };
  int group = 0, ahead = 0;
  const int tiles = 12;
  std::vector<bool> swept(tiles + 1);
  for (int n = 0; n <= tiles; n++) swept[n] = n < tiles && std::rand() % 5 != 0;
  for (int n = 0; n < tiles; n++) {
    if (!swept[n]) {
      group += NG;
      ahead = 0;
      continue;
    }
    auto id = [&](int t, int d) { return (long)t * 100000 + d; };
    if (ahead < std::min(DG, NG)) {
      const bool first = n == 0;
      for (; ahead < std::min(DG, NG); ahead++)
        for (int i = 0; i < 4; i++) {
          const int d = 4 * ahead + i;
          if (d < NC || fill)
            if (int e = write((4 * (group + ahead) + i) & (D - 1), d < NC ? id(n, d) : -1)) return e;
          if (first) commits++;
        }
      if (first) {
        commits = D;
      } else {
        commits++;
        landed = commits;
      }
    }
    ahead = 0;
    const int known_at = std::rand() % (NG + 2);  // the group from which on the next ticket is out
    for (int gi = 0; gi < NG; gi++) {
      const bool known = gi >= known_at && swept[n + 1];
      const sc::SweepAhead go = sc::sweep_ahead(gi, NC, DG, ahead, known);
      if (go.next && go.chunks) ahead++;
      for (int i = 0; i < 4; i++) {
        const int d = 4 * gi + i, s = (4 * group + i) & (D - 1);
        if (d < NC) {
          landed = std::max(landed, commits - (D - 1));
          if (slot[s].chunk != id(n, d) || slot[s].commit >= landed) return 3;
          slot[s].read = true;
        }
        if (i < go.chunks || fill)
          if (int e = write(s, i < go.chunks ? id(go.next ? n + 1 : n, 4 * go.group + i) : -1)) return e;
        commits++;
      }
      group++;
    }
  }
  return 0;
}
int main() {
  int caught = 0;
  for (int D : {4, 8})
    for (int NC = 3; NC < 80; NC++)
      for (unsigned seed = 1; seed < 60; seed++) {
        if (int e = play(D, NC, seed, false)) {
          std::printf("FAIL %d: D %d NC %d seed %u\n", e, D, NC, seed);
          return 1;
        }
        caught += play(D, NC, seed, true) == 1;
      }
  std::printf(caught ? "ok\n" : "the zero fill was not caught\n");
  return caught ? 0 : 1;
}
'''


def test_no_stage_slot_gets_a_copy_before_its_last_one_landed(tmp_path):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc) and shutil.which(nvcc) is None:
        pytest.skip("no nvcc")
    src = tmp_path / "stages.cu"
    src.write_text("#pragma nv_diag_suppress 177\n" + _SRC)
    exe = tmp_path / "stages"
    subprocess.check_call([nvcc, "-std=c++17", "-O1", "-ccbin", "g++", "--expt-relaxed-constexpr", "-gencode",
                           "arch=compute_100a,code=sm_100a", "-I", os.path.join(ROOT, "simcraft_b200", "csrc"), str(src),
                           "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
