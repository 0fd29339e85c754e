"""The ticket words of the sweeps (sc_sweep.cuh) on the CPU: every tile of a grid comes
back from its word, with its bits, also where a grid has more than 4096 tiles along x
or y (65,536 cells in x, 32,768 in y), and no tile's word says that there is none."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_SRC = r'''
#pragma nv_diag_suppress 177
#include <cstdio>
#include "sc_sweep.cuh"
using sc::SweepLayout;
int main() {
  const int dims[][3] = {{16, 8, 4},       {65536, 8, 1},  {65552, 8, 1}, {65552, 17, 2}, {5, 40000, 1},
                         {200, 32776, 1}, {1 << 20, 9, 1}, {3, 1 << 22, 1}, {4096, 4096, 1}};
  const int shapes[][2] = {{1, 1}, {1, 2}, {2, 4}, {4, 4}, {16, 1}, {1, 16}};
  for (const auto& d : dims)
    for (const auto& c : shapes) {
      const SweepLayout g = SweepLayout::make(d[0], d[1], d[2]);
      if (g.ntiles() > sc::kMaxTiles) return 1;
      for (int uy = 0; uy * c[1] < g.nty; uy++)
        for (int ux = 0; ux * c[0] < g.ntx; ux++)
          for (int r = 0; r < c[0] * c[1]; r++) {
            const int X = ux * c[0] + r % c[0], Y = uy * c[1] + r / c[0];
            const bool in = X < g.ntx && Y < g.nty;
            for (unsigned bits : {0u, 16u, 21u, 31u}) {
              if (!in && bits) continue;  // a tile outside the grid is not swept
              const unsigned w = sc::ticket_pack(g, c[0], c[1], make_int2(ux, uy), r, bits);
              if (w == sc::kNoTile || sc::ticket_bits(w) != (int)bits || (bits && sc::ticket_tile(w) != Y * g.ntx + X)) {
                std::printf("FAIL %d %d %d, shape %d %d, tile %d %d bits %u: word %x\n", d[0], d[1], d[2], c[0], c[1], X, Y,
                            bits, w);
                return 1;
              }
            }
          }
    }
  // the last tile that a grid may have
  SweepLayout g{};
  g.ntx = sc::kMaxTiles;
  g.nty = 1;
  const unsigned w = sc::ticket_pack(g, 1, 1, make_int2(sc::kMaxTiles - 1, 0), 0, 31);
  if (w == sc::kNoTile || sc::ticket_tile(w) != sc::kMaxTiles - 1 || sc::ticket_bits(w) != 31) return 1;
  std::printf("ok\n");
  return 0;
}
'''


def test_every_tile_comes_back_from_its_ticket_word(tmp_path):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc) and shutil.which(nvcc) is None:
        pytest.skip("no nvcc")
    src = tmp_path / "tickets.cu"
    src.write_text(_SRC)
    exe = tmp_path / "tickets"
    subprocess.check_call([nvcc, "-std=c++17", "-O1", "-ccbin", "g++", "--expt-relaxed-constexpr", "-gencode",
                           "arch=compute_100a,code=sm_100a", "-I", os.path.join(ROOT, "simcraft_b200", "csrc"), str(src),
                           "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
