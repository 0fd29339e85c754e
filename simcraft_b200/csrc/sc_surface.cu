// sc_surface.cu -- marching cubes (rebuildSurface, FluidSim/src/cpu/rebuild-surface.cc:686-741).
//
// The reference walks the (nx+1)(ny+1)(nz+1) cubes serially and numbers each
// vertex the first time a cube meets its edge, through a hash map.  Here the
// numbering is recomputed in parallel (sc_surface_dev.cuh): each cube creates
// the vertices of its crossing edges among {5, 6, 10}, and exclusive scans of
// the per-cube vertex and index counts, in the reference's cube order, place
// every vertex and index entry where the serial loop puts it.
//
//   k_mc_count     one pass over the SDF: case mask per cube (1 byte), per-block
//                  totals of vertices and index entries
//   k_mc_scan      one block: exclusive scan of the block totals, grand totals
//   k_mc_vertices  one scan per block over its cubes' vertex counts; writes each
//                  creating cube's first vertex number, and the block's vertices
//                  from a list in shared memory
//   k_mc_indices   the same for the index entries, over a list of the crossing cubes;
//                  each entry is the owner cube's first vertex number plus the edge's
//                  rank in its case
//
// Blocks own contiguous runs of kChunk cubes.  A few percent of the cubes cross the
// surface, so a thread per cube left one or two lanes of a warp in the long FP64 part
// (192^3: vertices 403 us, indices 241 us, with 16 block scans of 256 cubes each): a
// thread now reads the masks of 16 consecutive cubes in one load, one scan places all
// of them, and the vertices and the crossing cubes are dense lists that all threads
// share.  What remains is HBM and L2: the SDF once (8 bytes per sample; a lane loads
// the four corners at its z and has the next four from its neighbour), the masks three
// times (1 byte per cube), and the mesh itself.
#include <string>

#include "sc_surface.cuh"
#include "sc_surface_dev.cuh"

namespace sc {
namespace {

constexpr int kThreads = 256;
constexpr int kPer = 16;
constexpr int64_t kChunk = (int64_t)kThreads * kPer;

// The cases and what the kernels need of each (mc::case_info), worked out by the
// compiler: in each block of the kernels it took most of their time.
__device__ const uint64_t d_mc_cases[256] = {SC_MC_CASES_INIT};
struct CaseInfos {
  uint32_t v[256];
};
constexpr CaseInfos make_case_infos() {
  constexpr uint64_t cases[256] = {SC_MC_CASES_INIT};
  CaseInfos t{};
  for (int m = 0; m < 256; m++) t.v[m] = mc::case_info(cases[m]);
  return t;
}
__device__ const CaseInfos d_mc_infos = make_case_infos();

// In shared memory: a warp's cubes index it divergently.
__device__ __forceinline__ void load_cases(uint32_t* s) {
  for (int m = threadIdx.x; m < 256; m += blockDim.x) s[m] = d_mc_infos.v[m];
  __syncthreads();
}

// Exclusive scan of one int per thread over the 256-thread block; *total gets
// the block's sum.  `sh` holds 8 ints; the trailing barrier lets the caller
// reuse it at once.
__device__ __forceinline__ int block_exclusive_scan(int v, int* total, int* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int s = lane < kThreads / 32 ? sh[lane] : 0;
#pragma unroll
    for (int o = 1; o < kThreads / 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < kThreads / 32) sh[lane] = s;
  }
  __syncthreads();
  const int before = warp ? sh[warp - 1] : 0;
  *total = sh[kThreads / 32 - 1];
  __syncthreads();
  return before + x - v;
}

struct Scratch {
  uint8_t* mask;       // per cube
  uint32_t* vbase;     // per cube: first vertex number (creating cubes only)
  longlong2* bsum;     // per block: (index entries, vertices), then their exclusive prefix
  long long* totals;   // (index entries, vertices)
  unsigned* status;    // 1: an index entry found no vertex
};

__host__ __device__ inline size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

Scratch carve(void* base, int64_t ncubes, int64_t nblocks) {
  char* p = (char*)base;
  Scratch s;
  s.mask = (uint8_t*)p;
  p += align256((size_t)ncubes);
  s.vbase = (uint32_t*)p;
  p += align256(sizeof(uint32_t) * (size_t)ncubes);
  s.bsum = (longlong2*)p;
  p += align256(sizeof(longlong2) * (size_t)nblocks);
  s.totals = (long long*)p;
  s.status = (unsigned*)(p + 2 * sizeof(long long));
  return s;
}

__global__ void __launch_bounds__(kThreads) k_mc_count(mc::Grid g, Scratch s) {
  __shared__ uint32_t cases[256];
  __shared__ long long red[2][kThreads / 32];
  load_cases(cases);
  const int64_t nc = g.ncubes(), base = blockIdx.x * kChunk;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // signs of the corners (x, y) = (i, j), (i, j + 1), (i + 1, j), (i + 1, j + 1) at z
  // (32-bit offsets: there are fewer than 2^31 cubes, and so samples; i runs past the
  // grid in a last block's cubes that do not exist)
  const int sx = g.ny * g.nz;
  auto corners = [&](int i, int j, int z) {
    const int o = (i * g.ny + j) * g.nz + z;
    const bool in = z >= 0 && z < g.nz, x0 = in && i >= 0 && i < g.nx, x1 = in && i + 1 < g.nx, y0 = j >= 0, y1 = j + 1 < g.ny;
    const double a = x0 && y0 ? __ldg(g.sdf + o) : 1.0, b = x0 && y1 ? __ldg(g.sdf + o + g.nz) : 1.0,
                 c = x1 && y0 ? __ldg(g.sdf + o + sx) : 1.0, d = x1 && y1 ? __ldg(g.sdf + o + sx + g.nz) : 1.0;
    return (a < 0.0 ? 1 : 0) | (b < 0.0 ? 2 : 0) | (c < 0.0 ? 4 : 0) | (d < 0.0 ? 8 : 0);
  };
  int nv = 0, ni = 0;
  const int64_t c0 = base + threadIdx.x;
  int i, j, k;
  g.cube(c0 < nc ? c0 : nc - 1, i, j, k);
  for (int r = 0; r < kPer; r += 4) {
    if (base + (int64_t)r * kThreads >= nc) break;  // uniform over the block
    int lo[4], up[4];
    bool top[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {  // four cubes' loads in flight
      lo[u] = corners(i, j, k);
      up[u] = lane == 31 ? corners(i, j, k + 1) : 0;
      top[u] = k == g.nz - 1;
      // kThreads cubes on
      for (k += kThreads; k >= g.nz;) {
        k -= g.nz + 1;
        if (++j >= g.ny) {
          j = -1;
          i++;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      // the next lane's cube is the next one along z, except behind a row's last cube,
      // whose upper corners lie outside the grid
      int hi = __shfl_down_sync(0xffffffffu, lo[u], 1);
      if (lane == 31) hi = up[u];
      if (top[u]) hi = 0;
      const int64_t c = c0 + (int64_t)(r + u) * kThreads;
      if (c < nc) {
        const int m = mc::Grid::mask_of(lo[u], hi);
        s.mask[c] = (uint8_t)m;
        const uint32_t w = cases[m];
        nv += mc::info_owned(w);
        ni += mc::info_entries(w);
      }
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    nv += __shfl_xor_sync(0xffffffffu, nv, o);
    ni += __shfl_xor_sync(0xffffffffu, ni, o);
  }
  if (lane == 0) {
    red[0][warp] = ni;
    red[1][warp] = nv;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long a = 0, b = 0;
    for (int q = 0; q < kThreads / 32; q++) {
      a += red[0][q];
      b += red[1][q];
    }
    s.bsum[blockIdx.x] = make_longlong2(a, b);
  }
}

// One block of 1024 threads: exclusive scan of the per-block totals in place.
__global__ void __launch_bounds__(1024) k_mc_scan(int64_t nb, Scratch s) {
  __shared__ long long sa[1024], sb[1024];
  __shared__ long long carry[2];
  if (threadIdx.x == 0) carry[0] = carry[1] = 0;
  __syncthreads();
  for (int64_t base = 0; base < nb; base += 1024) {
    const int64_t q = base + threadIdx.x;
    const longlong2 v = q < nb ? s.bsum[q] : make_longlong2(0, 0);
    sa[threadIdx.x] = v.x;
    sb[threadIdx.x] = v.y;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      const long long ta = threadIdx.x >= o ? sa[threadIdx.x - o] : 0;
      const long long tb = threadIdx.x >= o ? sb[threadIdx.x - o] : 0;
      __syncthreads();
      sa[threadIdx.x] += ta;
      sb[threadIdx.x] += tb;
      __syncthreads();
    }
    if (q < nb) s.bsum[q] = make_longlong2(carry[0] + sa[threadIdx.x] - v.x, carry[1] + sb[threadIdx.x] - v.y);
    __syncthreads();
    if (threadIdx.x == 1023) {
      carry[0] += sa[1023];
      carry[1] += sb[1023];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    s.totals[0] = carry[0];
    s.totals[1] = carry[1];
    *s.status = 0;
  }
}

// The masks of a thread's kPer consecutive cubes (zero beyond the last cube).
struct Masks {
  uint32_t w[kPer / 4];
  __device__ __forceinline__ int operator[](int q) const { return (int)(w[q >> 2] >> 8 * (q & 3) & 0xffu); }
};
__device__ __forceinline__ Masks load_masks(const uint8_t* mask, int64_t c, int64_t nc) {
  static_assert(kPer == 16, "one 16-byte load");
  Masks m{};
  if (c + kPer <= nc) {
    const uint4 v = *reinterpret_cast<const uint4*>(mask + c);
    m.w[0] = v.x, m.w[1] = v.y, m.w[2] = v.z, m.w[3] = v.w;
  } else {
    for (int q = 0; q < kPer; q++)
      if (c + q < nc) m.w[q >> 2] |= (uint32_t)mask[c + q] << 8 * (q & 3);
  }
  return m;
}

__global__ void __launch_bounds__(kThreads) k_mc_vertices(mc::Grid g, Scratch s, double* V, double* N) {
  __shared__ uint32_t cases[256];
  __shared__ int sh[kThreads / 32];
  __shared__ uint16_t items[3 * kChunk];  // the block's vertices: cube (12 bits), owned edge (2 bits)
  load_cases(cases);
  const int64_t nc = g.ncubes(), base = blockIdx.x * kChunk, c0 = base + threadIdx.x * kPer;
  const long long next = s.bsum[blockIdx.x].y;
  const Masks m = load_masks(s.mask, c0, nc);
  int cnt = 0;
#pragma unroll
  for (int q = 0; q < kPer; q++) cnt += mc::info_owned(cases[m[q]]);
  int total;
  int at = block_exclusive_scan(cnt, &total, sh);
  if (cnt)
    for (int q = 0; q < kPer; q++) {
      const uint32_t w = cases[m[q]];
      const int n = mc::info_owned(w);
      if (!n) continue;
      s.vbase[c0 + q] = (uint32_t)(next + at);
      for (int o = 0; o < 3; o++) {
        const int r = mc::info_rank(w, o);
        if (r < n) items[at + r] = (uint16_t)((threadIdx.x * kPer + q) | o << 12);
      }
      at += n;
    }
  __syncthreads();
  for (int v = threadIdx.x; v < total; v += kThreads) {
    const int it = items[v];
    int i, j, k;
    g.cube(base + (it & 4095), i, j, k);
    double p[3], n[3];
    g.vertex(i, j, k, mc::owned_edge(it >> 12), p, n);
    for (int d = 0; d < 3; d++) {
      V[3 * (next + v) + d] = p[d];
      N[3 * (next + v) + d] = n[d];
    }
  }
}
static_assert(kChunk == 4096, "a cube's number within its block fits 12 bits");

__global__ void __launch_bounds__(kThreads) k_mc_indices(mc::Grid g, Scratch s, uint32_t* I) {
  __shared__ uint32_t cases[256];
  __shared__ int sh[kThreads / 32];
  __shared__ uint16_t cube[kChunk], first[kChunk];  // the block's crossing cubes and their first entries
  __shared__ uint64_t table[256];
  for (int q = threadIdx.x; q < 256; q += kThreads) table[q] = d_mc_cases[q];
  load_cases(cases);
  const int64_t nc = g.ncubes(), base = blockIdx.x * kChunk, c0 = base + threadIdx.x * kPer;
  const long long next = s.bsum[blockIdx.x].x;
  const Masks m = load_masks(s.mask, c0, nc);
  // crossing cubes (at most 4096) above, their entries (at most 15 each) below
  int cnt = 0;
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const int n = mc::info_entries(cases[m[q]]);
    cnt += n ? (1 << 17) + n : 0;
  }
  int total;
  int at = block_exclusive_scan(cnt, &total, sh);
  if (cnt)
    for (int q = 0; q < kPer; q++) {
      const int n = mc::info_entries(cases[m[q]]);
      if (!n) continue;
      cube[at >> 17] = (uint16_t)(threadIdx.x * kPer + q);
      first[at >> 17] = (uint16_t)(at & 0x1ffff);
      at += (1 << 17) + n;
    }
  __syncthreads();
  bool ok = true;
  for (int a = threadIdx.x; a < total >> 17; a += kThreads) {
    const int64_t c = base + cube[a];
    int i, j, k;
    g.cube(c, i, j, k);
    ok &= mc::emit_entries(g, i, j, k, table[s.mask[c]], [&](int mk, int oe) { return mc::info_find(cases[mk], oe); },
                           s.mask, s.vbase, next + first[a], I);
  }
  if (!ok) atomicOr(s.status, 1u);
}

mc::Grid to_grid(const SurfaceArgs& a) {
  return mc::Grid{a.nx, a.ny, a.nz, a.hx, a.hy, a.hz, a.ox, a.oy, a.oz, a.sdf};
}

int64_t nblocks(const mc::Grid& g) { return (g.ncubes() + kChunk - 1) / kChunk; }

}  // namespace

size_t surface_scratch_bytes(const SurfaceArgs& a) {
  const mc::Grid g = to_grid(a);
  const int64_t nc = g.ncubes();
  return align256((size_t)nc) + align256(sizeof(uint32_t) * (size_t)nc) +
         align256(sizeof(longlong2) * (size_t)nblocks(g)) + 256;
}

int surface_count(cudaStream_t st, const SurfaceArgs& a, void* scratch, int64_t* nvertices,
                  int64_t* nindices) {
  const mc::Grid g = to_grid(a);
  const int64_t nb = nblocks(g);
  const Scratch s = carve(scratch, g.ncubes(), nb);
  k_mc_count<<<(unsigned)nb, kThreads, 0, st>>>(g, s);
  k_mc_scan<<<1, 1024, 0, st>>>(nb, s);
  long long tot[2] = {0, 0};
  cudaMemcpyAsync(tot, s.totals, sizeof(tot), cudaMemcpyDeviceToHost, st);
  if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess) return -2;
  *nindices = tot[0];
  *nvertices = tot[1];
  return 0;
}

int surface_fill(cudaStream_t st, const SurfaceArgs& a, void* scratch, double* vertices, double* normals,
                 uint32_t* indices, std::string* msg) {
  const mc::Grid g = to_grid(a);
  const int64_t nb = nblocks(g);
  const Scratch s = carve(scratch, g.ncubes(), nb);
  k_mc_vertices<<<(unsigned)nb, kThreads, 0, st>>>(g, s, vertices, normals);
  k_mc_indices<<<(unsigned)nb, kThreads, 0, st>>>(g, s, indices);
  unsigned status = 0;
  cudaMemcpyAsync(&status, s.status, sizeof(status), cudaMemcpyDeviceToHost, st);
  if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess) return -2;
  if (status) {
    if (msg) *msg = "rebuild_surface: an index entry found no vertex";
    return -1;
  }
  return 0;
}

}  // namespace sc
