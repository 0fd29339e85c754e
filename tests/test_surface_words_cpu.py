"""What the surface kernels run (sc_surface_dev.cuh), built as host C++: the packed word of
each of the 256 cases says what the case itself says, a mask put together from the signs
of four lower and four upper corners is the cube's mask, and the kernels' route (lists of
vertices by owned edge, entries by the words) gives the mesh that the plain per-cube
functions give, which test_surface_cpu.py pins to the oracle."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_SRC = r'''
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "sc_surface_dev.cuh"
using namespace sc::mc;
static const uint64_t kCases[256] = {SC_MC_CASES_INIT};
struct Cases { uint64_t operator()(int m) const { return kCases[m]; } };
#define CHECK(c) do { if (!(c)) { std::printf("FAIL %s at line %d\n", #c, __LINE__); return 1; } } while (0)
static int words() {
  for (int m = 0; m < 256; m++) {
    const uint64_t w = kCases[m];
    const uint32_t v = case_info(w);
    CHECK(info_entries(v) == (int)SC_MC_COUNT(w));
    CHECK(info_owned(v) == owned_count(w));
    int seen = 0;
    for (int o = 0; o < 3; o++) {
      const int e = owned_edge(o), r = owned_rank(w, e);
      CHECK(owned(e) && info_find(v, e) == r && info_rank(v, o) == (r < 0 ? 3 : r));
      if (r >= 0) seen |= 1 << r;
    }
    CHECK(seen == (1 << owned_count(w)) - 1);  // the ranks are 0 .. count - 1
    int lo = 0, hi = 0;
    for (int c = 0; c < 8; c++)
      if (m >> c & 1) (SC_MC_CORNER_Z(c) ? hi : lo) |= 1 << (2 * SC_MC_CORNER_X(c) + SC_MC_CORNER_Y(c));
    CHECK(Grid::mask_of(lo, hi) == m);
  }
  return 0;
}
static int mesh(int nx, int ny, int nz, int special) {
  std::vector<double> sdf((size_t)nx * ny * nz);
  for (double& s : sdf) {
    s = std::rand() / (double)RAND_MAX - 0.5;
    const int q = std::rand() % 20;
    if (special && q < 4) s = q == 0 ? NAN : q == 1 ? INFINITY : q == 2 ? -INFINITY : -0.0;
  }
  const Grid g{nx, ny, nz, 0.1, 0.2, 0.3, -1.0, 0.5, 2.0, sdf.data()};
  const int64_t nc = g.ncubes();
  std::vector<uint8_t> mask(nc);
  std::vector<uint32_t> vbase(nc, 0xffffffffu), vbase2(nc, 0xffffffffu);
  std::vector<int64_t> ibase(nc);
  std::vector<std::pair<int64_t, int>> items;
  int64_t nv = 0, ni = 0;
  auto signs = [&](int i, int j, int z) {  // the four corners at z
    int s = 0;
    for (int a = 0; a < 2; a++)
      for (int b = 0; b < 2; b++) s |= (g.eval(i + a, j + b, z) < 0.0) << (2 * a + b);
    return s;
  };
  for (int64_t c = 0; c < nc; c++) {
    int i, j, k;
    g.cube(c, i, j, k);
    CHECK(g.cube_index(i, j, k) == c);
    mask[c] = (uint8_t)Grid::mask_of(signs(i, j, k), signs(i, j, k + 1));
    CHECK(mask[c] == g.mask(i, j, k));
    const uint64_t w = kCases[mask[c]];
    const uint32_t v = case_info(w);
    ibase[c] = ni;
    if (owned_count(w)) vbase[c] = (uint32_t)nv;
    const int n = info_owned(v);
    if (n) vbase2[c] = (uint32_t)nv;
    items.resize(nv + n);
    for (int o = 0; o < 3; o++)
      if (info_rank(v, o) < n) items[nv + info_rank(v, o)] = {c, o};
    nv += n;
    ni += info_entries(v);
  }
  CHECK(vbase == vbase2);
  std::vector<double> V(3 * nv), N(3 * nv), V2(3 * nv), N2(3 * nv);
  std::vector<uint32_t> I(ni), I2(ni);
  for (int64_t c = 0; c < nc; c++) {
    int i, j, k;
    g.cube(c, i, j, k);
    const uint64_t w = kCases[mask[c]];
    if (vbase[c] != 0xffffffffu) emit_vertices(g, i, j, k, w, vbase[c], V.data(), N.data());
    CHECK(emit_indices(g, i, j, k, w, Cases(), mask.data(), vbase.data(), ibase[c], I.data()));
    CHECK(emit_entries(g, i, j, k, w, [&](int m, int e) { return info_find(case_info(kCases[m]), e); }, mask.data(),
                       vbase.data(), ibase[c], I2.data()));
  }
  for (int64_t v = 0; v < nv; v++) {
    int i, j, k;
    g.cube(items[v].first, i, j, k);
    g.vertex(i, j, k, owned_edge(items[v].second), V2.data() + 3 * v, N2.data() + 3 * v);
  }
  CHECK(I == I2);
  CHECK(nv == 0 || (!std::memcmp(V.data(), V2.data(), 24 * nv) && !std::memcmp(N.data(), N2.data(), 24 * nv)));
  return 0;
}
int main() {
  std::srand(5);
  if (words()) return 1;
  const int dims[][3] = {{1, 1, 1}, {1, 4, 2}, {5, 6, 7}, {16, 15, 17}, {3, 40, 1}};
  for (const auto& d : dims)
    for (int special = 0; special < 2; special++)
      for (int r = 0; r < 4; r++)
        if (mesh(d[0], d[1], d[2], special)) return 1;
  std::printf("ok\n");
  return 0;
}
'''


def test_case_words_and_the_kernels_route(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "words.cc"
    src.write_text(_SRC)
    exe = tmp_path / "words"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-Wall", "-Werror", "-I",
                           os.path.join(ROOT, "simcraft_b200", "csrc"), str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
