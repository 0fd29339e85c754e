"""SweepLayout (sc_common.cuh) on the CPU, compiled as host code: off() is one to one
within the allocated elements for both element sizes, a lane's values of four steps
are whole 16-byte vectors of one 128-element chunk, and neighbouring cells within a
warp tile are adjacent lanes one step apart."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_SRC = r'''
#include <cstdio>
#include <vector>
#include "sc_common.cuh"
using sc::SweepLayout;
#define CHECK(c) do { if (!(c)) { std::printf("FAIL %s at line %d (%d %d %d)\n", #c, __LINE__, nx, ny, nz); return 1; } } while (0)
template <class T>
int run(int nx, int ny, int nz) {
  const SweepLayout g = SweepLayout::make(nx, ny, nz);
  CHECK(g.nc * 4 >= nz + 10);
  CHECK(g.total == (int64_t)g.ntiles() * 4 * g.nc * 128);
  std::vector<char> seen(g.total, 0);
  for (int x = 0; x < nx; x++)
    for (int y = 0; y < ny; y++)
      for (int z = 0; z < nz; z++) {
        const int64_t e = g.off<T>(x, y, z);
        CHECK(e >= 0 && e < g.total && !seen[e]);
        seen[e] = 1;
        const int sigma = z + (x & 7) + (y & 3), lane = (y & 3) * 8 + (x & 7);
        const int64_t chunk = e / 128;
        CHECK(chunk == g.chunk0(x / 16, y / 8, (y / 4 % 2) * 2 + x / 8 % 2) + sigma / 4);
        CHECK(e % 128 == SweepLayout::within<T>(sigma % 4, lane));
        // array a of a stream of n: the same place in chunk n * chunk + a
        CHECK(g.off<T>(x, y, z, 6, 2) == (chunk * 6 + 2) * 128 + e % 128);
      }
  constexpr int VE = 16 / (int)sizeof(T);
  for (int lane = 0; lane < 32; lane++)
    for (int s = 0; s < 4; s++) {
      const int w = SweepLayout::within<T>(s, lane);
      CHECK(w >= 0 && w < 128 && w / VE == s / VE * 32 + lane && w % VE == s % VE);
    }
  return 0;
}
int main() {
  const int sizes[][3] = {{1, 1, 1}, {8, 4, 1}, {9, 5, 2}, {17, 9, 13}, {16, 8, 32}, {33, 20, 7}, {31, 7, 6}};
  for (const auto& s : sizes)
    if (run<float>(s[0], s[1], s[2]) || run<double>(s[0], s[1], s[2])) return 1;
  std::printf("ok\n");
  return 0;
}
'''


def test_sweep_layout_index_arithmetic(tmp_path):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc) and shutil.which(nvcc) is None:
        pytest.skip("no nvcc")
    src = tmp_path / "layout.cu"
    src.write_text(_SRC)
    exe = tmp_path / "layout"
    subprocess.check_call([nvcc, "-std=c++17", "-O1", "-ccbin", "g++", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                           os.path.join(ROOT, "simcraft_b200", "csrc"), str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
