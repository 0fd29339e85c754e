// sc_pcg.cu -- MIC(0)-PCG pressure solver on B200 (sm_100a).
//
// Restates, on the GPU, the reference's CgSolver3D::solve
// (FluidSim/src/cpu/project-solver.cc:308-346), applyCompressedMatrix (:16-39),
// ModifiedIncompleteCholesky3D::precond (:230-306) and the masked BLAS-1 of
// FluidSim/src/cpu/util.cc:380-410.  The preconditioner's arithmetic is the
// reference's own (its non-standard pivot recurrence included); only the
// evaluation order changes: the lexicographic sweeps become i+j+k wavefronts.
//
// Structure of one PCG iteration (all kernels read their scalars from device
// memory, so a chunk of iterations is captured once as a CUDA graph):
//   k_spmv   Az = A s, partial s.Az          -> alpha      (project-solver.cc:328-331)
//   k_axpy   p += alpha s, r -= alpha Az     -> residual   (:332-335)
//   k_sweep  forward sweep  q = K^-1 r                     (:276-288)
//   k_sweep  backward sweep z = K^-T q, z.r -> beta        (:293-305, :338-341)
//   k_sa     s = z + beta s                  -> iter++     (:342, util.cc:404-410)
// The MIC(0) pivots E = 1/sqrt(e) are computed once per solve by a wavefront
// kernel; the reference recomputes them on every call with identical values.
//
// Two layouts.  The system as its producers write it (matrix, right-hand side,
// active flags, the pressure handed back, and the mixed solve's FP64 residual) is
// in the Tiled layout; the factors and the vectors of an iteration are in the
// SweepLayout, in which the sweeps (sc_sweep.cuh) stream whole chunks.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <type_traits>
#include <utility>
#include <vector>

#include <mutex>
#include <string>

#include "sc_sweep.cuh"

namespace sc {
namespace {

constexpr int kThreads = 256;
// 1: the iterations sweep only the tiles holding an active cell; 0: every tile
#ifndef SC_SKIP_EMPTY_TILES
#define SC_SKIP_EMPTY_TILES 1
#endif

enum { FIN_NONE = 0, FIN_INIT, FIN_SPMV, FIN_AXPY, FIN_BWD, FIN_SA, FIN_NORMS, FIN_EINIT, FIN_EAXPY, FIN_EREPLACE };

__device__ void finalize(int kind, PcgScalars* sc, double sum, double mx) {
  switch (kind) {
    case FIN_INIT: {  // r = rhs; residual check before the first preconditioner (:313-319)
      sc->rn2 = sum;
      sc->rinf = mx;
      sc->bnorm = sqrt(sum);
      double res = sc->criterion == CRIT_REL_L2 ? (sc->bnorm > 0.0 ? 1.0 : 0.0) : mx;
      sc->res = res;
      sc->first = 1;
      if (!isfinite(sum) || !(res == res)) {  // NaN/Inf in the right-hand side
        sc->err |= DEV_ERR_NONFINITE;
        sc->done = DONE_BREAKDOWN;
        sc->iter = 0;
      } else if (res < sc->tol) {
        sc->done = DONE_CONVERGED;
        sc->iter = 0;
      } else {
        sc->done = DONE_RUNNING;
        sc->iter = 1;
      }
      break;
    }
    case FIN_SPMV: {  // alpha = sigma / (s . z)  (:329-331)
      sc->sdotz = sum;
      if (sum == 0.0 || !isfinite(sum)) {
        sc->err |= (sum == 0.0) ? DEV_ERR_BREAKDOWN : DEV_ERR_NONFINITE;
        sc->done = DONE_BREAKDOWN;
      } else {
        sc->alpha = sc->sigma / sum;
      }
      break;
    }
    case FIN_AXPY: {  // residual = LinfNorm(r) (or relative L2); break when < tol (:334-335)
      sc->rn2 = sum;
      sc->rinf = mx;
      double res = sc->criterion == CRIT_REL_L2 ? (sc->bnorm > 0.0 ? sqrt(sum) / sc->bnorm : 0.0)
                                                : mx;
      sc->res = res;
      if (!isfinite(res)) {
        sc->err |= DEV_ERR_NONFINITE;
        sc->done = DONE_BREAKDOWN;
      } else if (res < sc->tol) {
        sc->done = DONE_CONVERGED;
      }
      break;
    }
    case FIN_BWD: {  // sigma_new = z . r ; beta = sigma_new / sigma (:338-341)
      if (sc->first) {
        sc->sigma = sum;
        sc->first = 0;
      } else {
        sc->beta = sum / sc->sigma;
        sc->sigma = sum;
      }
      if (!isfinite(sum)) {
        sc->err |= DEV_ERR_NONFINITE;
        sc->done = DONE_BREAKDOWN;
      }
      break;
    }
    case FIN_SA: {  // for-loop increment and bound (:327)
      sc->iter += 1;
      if (sc->iter >= sc->max_iter) sc->done = DONE_MAXITER;
      break;
    }
    case FIN_NORMS: {
      sc->rn2 = sum;
      sc->rinf = mx;
      break;
    }
    // Eisenstat iteration (FP32 inner solve): the residual of the split system is
    // rh = L^-1 r, rho = rh.rh = r.M^-1 r plays sigma's part and the stopping
    // measure is ||rh|| / ||rh_0||.
    case FIN_EINIT: {  // rho_0 = rh_0.rh_0 ; the first search direction is rh_0 (beta = 0)
      sc->sigma = sum;
      sc->beta = 0.0;
      sc->bnorm = sqrt(sum);
      sc->first = 0;
      if (!isfinite(sum)) {
        sc->err |= DEV_ERR_NONFINITE;
        sc->done = DONE_BREAKDOWN;
      } else if (sum == 0.0 && sc->done == DONE_RUNNING) {
        sc->done = DONE_CONVERGED;
        sc->iter = 0;
      }
      break;
    }
    case FIN_EREPLACE: {  // rh replaced by L^-1 of the FP64 residual: rho = rh.rh
      sc->sigma = sum;
      sc->res = sc->bnorm > 0.0 ? sqrt(sum) / sc->bnorm : 0.0;
      if (!isfinite(sum)) {
        sc->err |= DEV_ERR_NONFINITE;
        sc->done = DONE_BREAKDOWN;
      }
      break;
    }
    case FIN_EAXPY: {  // rho_new; convergence; beta = rho_new / rho
      sc->rn2 = sum;
      sc->rinf = mx;
      const double res = sc->bnorm > 0.0 ? sqrt(sum) / sc->bnorm : 0.0;
      sc->res = res;
      if (!isfinite(res)) {
        sc->err |= DEV_ERR_NONFINITE;
        sc->done = DONE_BREAKDOWN;
      } else if (res < sc->tol) {
        sc->done = DONE_CONVERGED;
      }
      sc->beta = sum / sc->sigma;
      sc->sigma = sum;
      break;
    }
    default:
      break;
  }
}

// Block reduce (sum, max) -> per-block partial -> last block reduces the
// partials in fixed order (deterministic) and runs the finalizer.
__device__ void reduce_finalize(double sum, double mx, double* partials, PcgScalars* sc,
                                int kind) {
  __shared__ double ss[32], sm[32];
  __shared__ bool last;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  sum = warp_sum(sum);
  mx = warp_max(mx);
  if (l == 0) {
    ss[w] = sum;
    sm[w] = mx;
  }
  __syncthreads();
  if (w == 0) {
    sum = l < nw ? ss[l] : 0.0;
    mx = l < nw ? sm[l] : 0.0;
    sum = warp_sum(sum);
    mx = warp_max(mx);
    if (l == 0) {
      partials[2 * blockIdx.x] = sum;
      partials[2 * blockIdx.x + 1] = mx;
      __threadfence();
      unsigned prev = atomicAdd(&sc->count, 1u);
      last = (prev == gridDim.x - 1);
    }
  }
  __syncthreads();
  if (last) {
    __threadfence();
    double s2 = 0.0, m2 = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
      s2 += __ldcg(&partials[2 * b]);
      m2 = fmax(m2, __ldcg(&partials[2 * b + 1]));
    }
    s2 = warp_sum(s2);
    m2 = warp_max(m2);
    __syncthreads();
    if (l == 0) {
      ss[w] = s2;
      sm[w] = m2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double S = 0.0, M = 0.0;
      for (int i = 0; i < nw; i++) {
        S += ss[i];
        M = fmax(M, sm[i]);
      }
      sc->count = 0;
      finalize(kind, sc, S, M);
      __threadfence();
    }
  }
}

// ---------------------------------------------------------------------------------
// Layout conversion (reference layout <-> tiled).  Row-block kernels: one
// 256-thread block owns the TY*32 elements of one (tile, slot) row block.
#define SC_ROWBLOCK_LOOP(g) \
  for (int rb = blockIdx.x, nrb_ = (g).ntiles() * (g).nz; rb < nrb_; rb += gridDim.x)

template <class Ts, class Td>
__global__ void __launch_bounds__(kThreads) k_to_tiled(Tiled g, const Ts* __restrict__ src,
                                                       Td* __restrict__ dst,
                                                       const uint8_t* __restrict__ mask_ref) {
  SC_ROWBLOCK_LOOP(g) {
    Cell c;
    c.init(g, rb, threadIdx.x);
    Td v = Td(0);
    if (c.inside) {
      const int64_t r = lin(c.x, c.y, c.z, g.ny, g.nz);
      if (!mask_ref || mask_ref[r]) v = (Td)src[r];
    }
    dst[c.e] = v;
  }
}
// An array of the system (axis 0, 1, 2: the couplings to the lower neighbour along x, y,
// z; -1: the diagonal).  Whole inactive rows and couplings to inactive cells are never
// read by applyCompressedMatrix (it tests the neighbour's activity first).  The SpMV and
// the pivots' products multiply them by zeros or use them as they are, so a non-finite
// value there becomes 0; finite values stay as given.
__global__ void __launch_bounds__(kThreads) k_matrix_to_tiled(Tiled g, const double* __restrict__ src, double* __restrict__ dst,
                                                              const uint8_t* __restrict__ act, int axis) {
  SC_ROWBLOCK_LOOP(g) {
    Cell c;
    c.init(g, rb, threadIdx.x);
    double v = 0.0;
    if (c.inside) {
      const int64_t r = lin(c.x, c.y, c.z, g.ny, g.nz);
      v = src[r];
      if (!isfinite(v)) {
        bool read = act[r];
        if (axis == 0) read = read && c.x > 0 && act[r - (int64_t)g.ny * g.nz];
        if (axis == 1) read = read && c.y > 0 && act[r - g.nz];
        if (axis == 2) read = read && c.z > 0 && act[r - 1];
        if (!read) v = 0.0;
      }
    }
    dst[c.e] = v;
  }
}
template <class Ts, class Td>
__global__ void __launch_bounds__(kThreads) k_from_tiled(Tiled g, const Ts* __restrict__ src,
                                                         Td* __restrict__ dst) {
  SC_ROWBLOCK_LOOP(g) {
    Cell c;
    c.init(g, rb, threadIdx.x);
    if (c.inside) dst[lin(c.x, c.y, c.z, g.ny, g.nz)] = (Td)src[c.e];
  }
}
template <class T>
__global__ void k_fill(int64_t n, T* __restrict__ dst, T v) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) dst[e] = v;
}

// max |A_Right(p) - A_Left(p+x)| (and Up/Down, Front/Back) over active pairs,
// the relation checkSystemSymmetry asserts (project-solver.cc:41-57).
__global__ void k_symmetry(int nx, int ny, int nz, const double* const* an,
                           const uint8_t* act, double* partials, PcgScalars* sc) {
  double mx = 0.0;
  const int64_t N = (int64_t)nx * ny * nz;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; id < N; id += stride) {
    if (!act[id]) continue;
    int k = (int)(id % nz);
    int j = (int)((id / nz) % ny);
    int i = (int)(id / ((int64_t)ny * nz));
    if (i < nx - 1 && act[id + (int64_t)ny * nz])
      mx = fmax(mx, fabs(an[1][id] - an[0][id + (int64_t)ny * nz]));
    if (j < ny - 1 && act[id + nz]) mx = fmax(mx, fabs(an[2][id] - an[3][id + nz]));
    if (k < nz - 1 && act[id + 1]) mx = fmax(mx, fabs(an[4][id] - an[5][id + 1]));
  }
  reduce_finalize(0.0, mx, partials, sc, FIN_NORMS);
}

// ---------------------------------------------------------------------------------
// Elementwise kernels over a SweepLayout.  A thread owns the four consecutive
// elements at 4 * i (a 16- or 32-byte vector).
template <class T>
struct __align__(16) Vec4 {
  T e[4];
};
template <class T>
__device__ __forceinline__ Vec4<T> vload(const T* p) {
  return *reinterpret_cast<const Vec4<T>*>(p);
}
template <class T>
__device__ __forceinline__ void vstore(T* p, const Vec4<T>& v) {
  *reinterpret_cast<Vec4<T>*>(p) = v;
}

// Position of a lane's chunk in the grid: (x, y) of its column and z of its step
// 4 * chunk; `inside`: the column lies in the grid.  A chunk's four steps are four
// consecutive z, those outside [0, nz) padding.
struct ChunkPos {
  int tile, lane, x, y, z0;
  bool inside;
  int64_t chunk;  // over the grid
  int64_t e;      // element of the first step in one array (chunk_load, chunk_store)
  // and in array `a` of a stream of `arrays`
  template <class T>
  __device__ __forceinline__ int64_t in_stream(int arrays, int a) const {
    return (chunk * arrays + a) * 128 + lane * (16 / (int)sizeof(T));
  }
};
template <class T>
__device__ __forceinline__ ChunkPos chunk_pos(const SweepLayout& g, int64_t i) {  // i: chunk * 32 + lane over the grid
  const int lane = (int)(i & 31);
  const unsigned c = (unsigned)(i >> 5), w = c / (unsigned)g.nc, ch = c - w * (unsigned)g.nc;
  const int tile = (int)(w >> 2), ww = (int)(w & 3);
  const int Y = tile / g.ntx, X = tile - Y * g.ntx, tx = lane & 7, ty = lane >> 3;
  ChunkPos p;
  p.tile = tile;
  p.chunk = c;
  p.lane = lane;
  p.x = X * 16 + (ww & 1) * 8 + tx;
  p.y = Y * 8 + (ww >> 1) * 4 + ty;
  p.z0 = (int)ch * 4 - tx - ty;
  p.inside = p.x < g.nx && p.y < g.ny;
  p.e = (int64_t)c * 128 + lane * (16 / (int)sizeof(T));
  return p;
}
#define SC_CHUNK_LOOP(i, g) \
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (g).total / 4; i += (int64_t)gridDim.x * blockDim.x)

// r = scale * src on active cells (src in the Tiled layout, r in the SweepLayout), p = 0.
template <class T>
__global__ void __launch_bounds__(kThreads) k_init(Tiled tg, SweepLayout g, const double* __restrict__ src,
                                                   double scale, const uint8_t* __restrict__ act,
                                                   T* __restrict__ r, T* __restrict__ p,
                                                   double* partials, PcgScalars* sc,
                                                   int fin = FIN_INIT) {
  double s2 = 0.0, mx = 0.0;
  SC_CHUNK_LOOP(i, g) {
    const ChunkPos c = chunk_pos<T>(g, i);
    T v[4], zero[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int z = c.z0 + j;
      v[j] = T(0);
      if (c.inside && z >= 0 && z < g.nz) {
        const int64_t o = tg.off(c.x, c.y, z);
        if (act[o]) v[j] = (T)(src[o] * scale);
      }
      const double dv = (double)v[j];
      s2 += dv * dv;
      mx = fmax(mx, fabs(dv));
    }
    chunk_store(r + c.e, v);
    chunk_store(p + c.e, zero);
  }
  reduce_finalize(s2, mx, partials, sc, fin);
}
// Norms of src on active cells, and (out given) its masked copy; Tiled layout.
__global__ void __launch_bounds__(kThreads) k_norms(int64_t n, const double* __restrict__ src,
                                                    const uint8_t* __restrict__ act, double* __restrict__ out,
                                                    double* partials, PcgScalars* sc) {
  double s2 = 0.0, mx = 0.0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
    const double v = act[e] ? src[e] : 0.0;
    if (out) out[e] = v;
    s2 += v * v;
    mx = fmax(mx, fabs(v));
  }
  reduce_finalize(s2, mx, partials, sc, FIN_NORMS);
}
// SweepLayout -> Tiled (the pressure handed back) and Tiled -> SweepLayout.
template <class T>
__global__ void __launch_bounds__(kThreads) k_sweep_to_tiled(SweepLayout g, Tiled tg, const T* __restrict__ src,
                                                             double* __restrict__ dst) {
  SC_ROWBLOCK_LOOP(tg) {
    Cell c;
    c.init(tg, rb, threadIdx.x);
    dst[c.e] = c.inside ? (double)src[g.off<T>(c.x, c.y, c.z)] : 0.0;
  }
}
// Reference layout <-> SweepLayout.
template <class T>
__global__ void __launch_bounds__(kThreads) k_ref_to_sweep(SweepLayout g, const double* __restrict__ src, T* __restrict__ dst) {
  SC_CHUNK_LOOP(i, g) {
    const ChunkPos c = chunk_pos<T>(g, i);
    T v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int z = c.z0 + j;
      v[j] = c.inside && z >= 0 && z < g.nz ? (T)src[lin(c.x, c.y, z, g.ny, g.nz)] : T(0);
    }
    chunk_store(dst + c.e, v);
  }
}
template <class T>
__global__ void __launch_bounds__(kThreads) k_sweep_to_ref(SweepLayout g, const T* __restrict__ src, double* __restrict__ dst) {
  SC_CHUNK_LOOP(i, g) {
    const ChunkPos c = chunk_pos<T>(g, i);
    const Quad<T> v = chunk_load(src + c.e);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int z = c.z0 + j;
      if (c.inside && z >= 0 && z < g.nz) dst[lin(c.x, c.y, z, g.ny, g.nz)] = (double)v.e[j];
    }
  }
}

// The iteration kernels below visit only the tiles of a sweep order list
// (tiles[-1].x entries; the tiles holding an active cell): the vectors they
// update are zero on every other tile and stay so.  Work unit: nc-th part of a
// tile, 512 consecutive elements, four per thread of half a block.
__device__ __forceinline__ int unit_count(const SweepLayout& g, const int2* __restrict__ tiles) {
  return tiles[-1].x * g.nc;
}
constexpr int kUnits = kThreads / 128;  // units a block visits at once
__device__ __forceinline__ int first_unit() { return blockIdx.x * kUnits + (threadIdx.x >> 7); }
__device__ __forceinline__ int64_t unit_elem(const SweepLayout& g, const int2* __restrict__ tiles, int c) {
  const int t = c / g.nc, u = c - t * g.nc;
  const int2 XY = tiles[t];
  return ((int64_t)(XY.y * g.ntx + XY.x) * g.nc + u) * 512 + 4 * (threadIdx.x & 127);
}

template <class T>
__global__ void __launch_bounds__(kThreads) k_copy(SweepLayout g, const int2* __restrict__ tiles, const T* __restrict__ a,
                                                   T* __restrict__ b, const PcgScalars* sc) {
  if (sc->done != DONE_RUNNING) return;
  const int nch = unit_count(g, tiles);
  for (int c = first_unit(); c < nch; c += kUnits * gridDim.x) {
    const int64_t e = unit_elem(g, tiles, c);
    vstore(b + e, vload(a + e));
  }
}

// applyCompressedMatrix (project-solver.cc:16-39) on the tiled layout.  The
// upper couplings come from the neighbours' lower ones (A symmetric,
// checkSystemSymmetry, :41-57).
// x(dx, dy, dz) is the vector's value at the cell's neighbour.
template <class X>
__device__ __forceinline__ double apply_row(const Tiled& g, const Cell& c, const double* __restrict__ adiag,
                                            const double* __restrict__ al, const double* __restrict__ ad,
                                            const double* __restrict__ ab, const uint8_t* __restrict__ act, X x) {
  const int64_t e = c.e;
  double t = adiag[e] * x(0, 0, 0);
  if (c.x > 0) {
    int64_t o = c.xm(g);
    if (act[o]) t += al[e] * x(-1, 0, 0);
  }
  if (c.y > 0) {
    int64_t o = c.ym(g);
    if (act[o]) t += ad[e] * x(0, -1, 0);
  }
  if (c.z > 0) {
    int64_t o = c.zm(g);
    if (act[o]) t += ab[e] * x(0, 0, -1);
  }
  if (c.x < g.nx - 1) {
    int64_t o = c.xp(g);
    if (act[o]) t += al[o] * x(1, 0, 0);
  }
  if (c.y < g.ny - 1) {
    int64_t o = c.yp(g);
    if (act[o]) t += ad[o] * x(0, 1, 0);
  }
  if (c.z < g.nz - 1) {
    int64_t o = c.zp(g);
    if (act[o]) t += ab[o] * x(0, 0, 1);
  }
  return t;
}

// The PCG's SpMV: the matrix as its producer wrote it (Tiled), x and y in the
// SweepLayout.  The vectors are zero on inactive cells, so only a row's own activity is
// tested.
// A block of 8 warps owns a 32 x 8 column tile (two sweep tiles) and walks a run of
// its slots: warp ty is row ty, and lane tx has cell z = (slot - tx) mod nz of its
// column, so that the z neighbours of a lane's cell are its own at the previous and
// next slot and the x neighbours the adjacent lanes' there.  A three-slot register
// window holds both (x by shuffle); the y neighbours are the adjacent rows at the
// same z, and only the two edge lanes of a row reach into the next tiles.  The matrix's
// rows of a slot are whole lines: from a copy of it in the SweepLayout, of whose 16-byte
// vectors a slot uses one element, FP64 took 1657 us at 512^3, now 1492 (4.41 TB/s).
// Every load is issued one slot ahead.  The upper couplings come from the neighbours' lower ones
// (A symmetric, checkSystemSymmetry, :41-57).
// The order in which a thread adds its products, and the tree that adds the threads'
// sums, decide the last bits of s.Az and with them the rounding of every later
// iterate: on systems whose MIC(0) factor is far from A (the tau terms), another
// order moved the FP64 solution by 2e-9 relative.  The walk is therefore part of the
// result, whatever the layout underneath.
template <class T>
__global__ void __launch_bounds__(kThreads, 3)
    k_spmv(SweepLayout g, Tiled tg, const int2* __restrict__ tiles, const T* __restrict__ adiag, const T* __restrict__ al,
           const T* __restrict__ ad, const T* __restrict__ ab, const uint8_t* __restrict__ act, const T* __restrict__ x,
           T* __restrict__ y, double* partials, PcgScalars* sc, int use_skip, int runs) {
  if (use_skip && sc->done != DONE_RUNNING) return;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int nz = g.nz;
  double acc = 0.0;
  const int items = tiles[-1].x * runs;
  // element of step sigma of a column: wb its warp tile's first element, ln its lane there
  auto at = [](int64_t wb, int sigma, int ln) { return wb + SweepLayout::within<T>(sigma, ln); };
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int li = it / runs, run = it - li * runs;
    const int s0 = (int)((int64_t)nz * run / runs), s1 = (int)((int64_t)nz * (run + 1) / runs);
    const int xg = tiles[li].x * 32 + tx, yg = tiles[li].y * 8 + ty;
    const bool inside = xg < g.nx && yg < g.ny;
    const bool hx = inside && xg > 0, px = inside && xg < g.nx - 1, hy = inside && yg > 0, py = inside && yg < g.ny - 1;
    // columns this lane reads: its own, the rows at y - 1 and y + 1 (read only when hy /
    // py), and for the edge lanes those at x - 1 and x + 1; outside the grid its own
    // stands in for padding that holds zeros, or for a column past the last tile
    auto column = [&](int X, int Y, int64_t& wb, int& ln, int& skew) {
      wb = g.chunk0(X >> 4, Y >> 3, ((Y >> 2) & 1) * 2 + ((X >> 3) & 1)) * 128;
      ln = (Y & 3) * 8 + (X & 7);
      skew = (Y & 3) + (X & 7);
    };
    const bool ex0 = tx == 0 && hx, ex31 = tx == 31 && px;
    int64_t wc, wym, wyp, wxe;
    int lc, lym, lyp, lxe, kc, kym, kyp, kxe;
    column(xg < g.ntx * 16 ? xg : xg - 16, yg, wc, lc, kc);
    column(xg < g.ntx * 16 ? xg : xg - 16, hy ? yg - 1 : yg, wym, lym, kym);
    column(xg < g.ntx * 16 ? xg : xg - 16, py ? yg + 1 : yg, wyp, lyp, kyp);
    column(ex0 ? xg - 1 : ex31 ? xg + 1 : (xg < g.ntx * 16 ? xg : xg - 16), yg, wxe, lxe, kxe);
    // the matrix: this lane's own row, the one at y + 1 in the same slot, and for the last
    // lane the first one of the next tile, whose slots are the z
    constexpr int RS = Tiled::TY * 32;
    const int64_t tb = tg.tile_base(tiles[li].x, tiles[li].y), row = tb + ty * 32 + tx,
                  ryp = ty < Tiled::TY - 1 ? row + 32 : tb + (int64_t)tg.ntx * tg.tile_elems + tx,
                  rxp = tb + tg.tile_elems + ty * 32;
    auto wrap = [nz](int v) { return v >= nz ? v - nz : v; };
    int sp = wrap(s0 + 1);  // the next slot
    int z = s0 - tx % nz;
    if (z < 0) z += nz;
    const int zm = z == 0 ? nz - 1 : z - 1;
    int zp = wrap(z + 1);
    T x_m = __ldg(x + at(wc, zm + kc, lc)), x_c = __ldg(x + at(wc, z + kc, lc)), x_p = __ldg(x + at(wc, zp + kc, lc));
    T al_c = __ldg(al + row + (int64_t)s0 * RS), al_p = __ldg(al + row + (int64_t)sp * RS);
    T ab_c = __ldg(ab + row + (int64_t)s0 * RS), ab_p = __ldg(ab + row + (int64_t)sp * RS);
    T d_n = __ldg(adiag + row + (int64_t)s0 * RS), adc_n = __ldg(ad + row + (int64_t)s0 * RS);
    uint8_t a_n = __ldg(act + row + (int64_t)s0 * RS);
    T ym_n = hy ? __ldg(x + at(wym, z + kym, lym)) : T(0), yp_n = py ? __ldg(x + at(wyp, z + kyp, lyp)) : T(0),
      adp_n = py ? __ldg(ad + ryp + (int64_t)s0 * RS) : T(0);
    T xe_n = ex0 || ex31 ? __ldg(x + at(wxe, z + kxe, lxe)) : T(0), ale_n = ex31 ? __ldg(al + rxp + (int64_t)z * RS) : T(0);
    for (int s = s0; s < s1; s++) {
      const int z2 = wrap(zp + 1), s2 = wrap(sp + 1);
      const T d = d_n, adc = adc_n, ymv = ym_n, ypv = yp_n, adp = adp_n, xe = xe_n, ale = ale_n;
      const bool a = inside && a_n;
      // the next window entries and the next slot's loads first: their latency
      // overlaps this slot's work
      const int64_t e1 = row + (int64_t)sp * RS, e2 = row + (int64_t)s2 * RS;
      const T x_n = __ldg(x + at(wc, z2 + kc, lc)), al_n = __ldg(al + e2), ab_n = __ldg(ab + e2);
      d_n = __ldg(adiag + e1);
      adc_n = __ldg(ad + e1);
      a_n = __ldg(act + e1);
      ym_n = hy ? __ldg(x + at(wym, zp + kym, lym)) : T(0);
      yp_n = py ? __ldg(x + at(wyp, zp + kyp, lyp)) : T(0);
      adp_n = py ? __ldg(ad + ryp + (int64_t)sp * RS) : T(0);
      xe_n = ex0 || ex31 ? __ldg(x + at(wxe, zp + kxe, lxe)) : T(0);
      ale_n = ex31 ? __ldg(al + rxp + (int64_t)zp * RS) : T(0);
      const bool hz = z > 0, pz = z < nz - 1;
      T xm = __shfl_up_sync(kFull, x_m, 1), xp = __shfl_down_sync(kFull, x_p, 1), alp = __shfl_down_sync(kFull, al_p, 1);
      if (tx == 0) xm = xe;
      if (tx == 31) {
        xp = xe;
        alp = ale;
      }
      const T cxm = hx ? al_c : T(0), cym = hy ? adc : T(0), czm = hz ? ab_c : T(0);
      const T cxp = px ? alp : T(0), cyp = py ? adp : T(0), czp = pz ? ab_p : T(0);
      T t = d * x_c;
      t += cxm * xm;
      t += cym * ymv;
      t += czm * x_m;
      t += cxp * xp;
      t += cyp * ypv;
      t += czp * x_p;
      const T o = a ? t : T(0);
      if (inside) y[at(wc, z + kc, lc)] = o;
      acc += (double)x_c * (double)o;
      x_m = x_c;
      x_c = x_p;
      x_p = x_n;
      al_c = al_p;
      al_p = al_n;
      ab_c = ab_p;
      ab_p = ab_n;
      z = zp;
      zp = z2;
      sp = s2;
    }
  }
  reduce_finalize(acc, 0.0, partials, sc, FIN_SPMV);
}

// b = A x with the reference's activity tests (x may be non-zero on inactive
// cells): applyCompressedMatrix for the apply entry point.  x and b in the
// reference layout.
__global__ void __launch_bounds__(kThreads)
    k_apply_checked(Tiled g, const double* __restrict__ adiag, const double* __restrict__ al,
                    const double* __restrict__ ad, const double* __restrict__ ab,
                    const uint8_t* __restrict__ act, const double* __restrict__ x, double* __restrict__ b) {
  SC_ROWBLOCK_LOOP(g) {
    Cell c;
    c.init(g, rb, threadIdx.x);
    if (!c.inside) continue;
    const int64_t r = lin(c.x, c.y, c.z, g.ny, g.nz);
    b[r] = act[c.e] ? apply_row(g, c, adiag, al, ad, ab, act,
                                [&](int dx, int dy, int dz) { return x[r + lin(dx, dy, dz, g.ny, g.nz)]; })
                    : 0.0;
  }
}

// saxpy(pg, s, alpha); saxpy(r, z, -alpha); residual (:332-335, util.cc:394-402).
// s and Az are zero on inactive cells, so the masked updates of the reference
// are the plain updates here.
template <class T>
__global__ void __launch_bounds__(kThreads)
    k_axpy(SweepLayout g, const int2* __restrict__ tiles, const T* __restrict__ s,
           const T* __restrict__ Az, T* __restrict__ p, T* __restrict__ r, double* partials,
           PcgScalars* sc, int fin = FIN_AXPY) {
  if (sc->done != DONE_RUNNING) return;
  const T alpha = (T)sc->alpha;
  double s2 = 0.0, mx = 0.0;
  const int nch = unit_count(g, tiles);
  for (int c = first_unit(); c < nch; c += kUnits * gridDim.x) {
    const int64_t e = unit_elem(g, tiles, c);
    const Vec4<T> sv = vload(s + e), av = vload(Az + e);
    Vec4<T> pv = vload(p + e), rv = vload(r + e);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      pv.e[k] = pv.e[k] + alpha * sv.e[k];
      rv.e[k] = rv.e[k] + (-alpha) * av.e[k];
      const double dv = (double)rv.e[k];
      s2 += dv * dv;
      mx = fmax(mx, fabs(dv));
    }
    vstore(p + e, pv);
    vstore(r + e, rv);
  }
  reduce_finalize(s2, mx, partials, sc, fin);
}

// scaleAndAdd(s, z, beta): s = z + beta s (util.cc:404-410); z and s are zero
// on inactive cells.
template <class T>
__global__ void __launch_bounds__(kThreads)
    k_sa(SweepLayout g, const int2* __restrict__ tiles, const T* __restrict__ z, T* __restrict__ s,
         double* partials, PcgScalars* sc) {
  if (sc->done != DONE_RUNNING) return;
  const T beta = (T)sc->beta;
  const int nch = unit_count(g, tiles);
  for (int c = first_unit(); c < nch; c += kUnits * gridDim.x) {
    const int64_t e = unit_elem(g, tiles, c);
    const Vec4<T> zv = vload(z + e);
    Vec4<T> sv = vload(s + e);
#pragma unroll
    for (int k = 0; k < 4; k++) sv.e[k] = zv.e[k] + beta * sv.e[k];
    vstore(s + e, sv);
  }
  reduce_finalize(0.0, 0.0, partials, sc, FIN_SA);
}

// The system in the SweepLayout, from the Tiled arrays: the diagonal and the
// lower couplings, zero in inactive rows and where they couple to an inactive
// cell (the reference never reads those), and the tau-weighted neighbour products
// of the pivot recurrence (project-solver.cc:244-265).  For the Left term these are
//   tau*A_L(p)*A_L(p-x+y) [if p-x+y active] + tau*A_L(p)*A_L(p-x+z) [if p-x+z active]
// and likewise for Down and Back; they only depend on A.  PivotOp uses a
// neighbour's terms only where that neighbour's pivot is not zero.  A coupling in
// these products may itself lead to an inactive cell and counts as it is given.
// tile_act (optional, zero on entry): 1 for the tiles holding an active cell.
// A thread has four cells of a column and reads them and the six columns around from
// each column's own base, all loads before they are used: testing each cell's activity
// first and looking up every element by its coordinates took 984 us at 256^3 (134 at
// 128^3), and a pass over the Tiled arrays that cleared the non-finite entries before
// that another 385 (57); now 480 (68) and none.
struct TiledColumn {
  int64_t base;
  int skew, nz;  // slot of z: (z + skew) mod nz
  __device__ __forceinline__ TiledColumn(const Tiled& g, int x, int y)
      : base(g.tile_base(x >> 5, y / Tiled::TY) + (y % Tiled::TY) * 32 + (x & 31)), skew((x & 31) % g.nz), nz(g.nz) {}
  __device__ __forceinline__ int64_t at(int z) const {  // z is moved into the grid
    const int s = min(max(z, 0), nz - 1) + skew;
    return base + (int64_t)(s >= nz ? s - nz : s) * (Tiled::TY * 32);
  }
};
__global__ void __launch_bounds__(kThreads, 2)
    k_sweep_system(SweepLayout g, Tiled tg, const double* __restrict__ adiag, const double* __restrict__ al,
                   const double* __restrict__ ad, const double* __restrict__ ab, const uint8_t* __restrict__ act,
                   double tau, PcgSolver::PivotIn out, uint8_t* __restrict__ tile_act) {
  SC_CHUNK_LOOP(i, g) {
    const ChunkPos c = chunk_pos<double>(g, i);
    double v[7][4] = {};
    bool any = false;
    if (c.inside && c.z0 + 3 >= 0 && c.z0 < g.nz) {
      const int x = c.x, y = c.y, z0 = c.z0;
      const bool hl = x > 0, hr = x < g.nx - 1, hd = y > 0, hu = y < g.ny - 1;
      // the cell's column and those around (the cell's own where there is none)
      const TiledColumn C(tg, x, y), L(tg, x - hl, y), R(tg, x + hr, y), D(tg, x, y - hd), U(tg, x, y + hu),
          LU(tg, x - (hl && hu), y + (hl && hu)), RD(tg, x + (hr && hd), y - (hr && hd));
      // bit j of a column: its cell at z0 - 1 + j is active
      auto active = [&](const TiledColumn& t, bool there, int from, int to) {
        unsigned bits = 0;
#pragma unroll
        for (int j = 0; j < 6; j++)
          if (j >= from && j <= to) bits |= (unsigned)(act[t.at(z0 - 1 + j)] != 0) << j;
        const unsigned in = 0x3fu & (z0 >= 1 ? ~0u : ~0u << (1 - z0)) & (z0 + 4 < g.nz ? ~0u : (1u << (g.nz - z0 + 1)) - 1u);
        return there ? bits & in : 0u;
      };
      const unsigned aC = active(C, true, 0, 4), aL = active(L, hl, 1, 5), aLU = active(LU, hl && hu, 1, 4),
                     aD = active(D, hd, 1, 5), aRD = active(RD, hr && hd, 1, 4), aR = active(R, hr, 0, 3),
                     aU = active(U, hu, 0, 3);
      any = (aC & 0x1eu) != 0;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int z = z0 + j;
        const int64_t e = C.at(z), eLz = L.at(z + 1), eDz = D.at(z + 1);
        const double d = adiag[e], l = al[e], dn = ad[e], b = ab[e];
        const double l1 = al[LU.at(z)], l2 = al[eLz], d1 = ad[RD.at(z)], d2 = ad[eDz], b1 = ab[R.at(z - 1)], b2 = ab[U.at(z - 1)];
        auto on = [&](unsigned bits, int at) { return (bits >> (j + 1 + at) & 1u) != 0; };
        if (!on(aC, 0)) continue;
        v[0][j] = d;
        if (on(aL, 0)) {
          v[1][j] = l;
          if (on(aLU, 0)) v[4][j] += tau * l * l1;
          if (on(aL, 1)) v[4][j] += tau * l * l2;
        }
        if (on(aD, 0)) {
          v[2][j] = dn;
          if (on(aRD, 0)) v[5][j] += tau * dn * d1;
          if (on(aD, 1)) v[5][j] += tau * dn * d2;
        }
        if (on(aC, -1)) {
          v[3][j] = b;
          if (on(aR, -1)) v[6][j] += tau * b * b1;
          if (on(aU, -1)) v[6][j] += tau * b * b2;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 7; k++) chunk_store(out.a[k] + c.e, v[k]);
    // a warp holds one chunk
    if (tile_act && __any_sync(kFull, any) && c.lane == 0) tile_act[c.tile] = 1;
  }
}

// The factor streams of a precision, from the FP64 forward stream the pivot sweep
// wrote (cL, cD, cB, E): the upper couplings in own-cell form for the backward
// sweep, uR(p) = cL(p+x) = A_L(p+x) E(p) etc. (the products of
// project-solver.cc:296-302), and in FP32 the forward stream with the diagonals of
// the Eisenstat operator, Pinv = 1/E and Dt = 2/E^2 - Adiag where E != 0, else 0.
template <class T>
__global__ void __launch_bounds__(kThreads)
    k_sweep_factor(SweepLayout g, const double* __restrict__ fwd64, const double* __restrict__ adiag, SysArrays<T> o) {
  constexpr int S = kFwdStream<double>;
  SC_CHUNK_LOOP(i, g) {
    const ChunkPos c = chunk_pos<T>(g, i);
    T b[4][4] = {}, f[6][4] = {};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int x = c.x, y = c.y, z = c.z0 + j;
      if (!c.inside || z < 0 || z >= g.nz) continue;
      const int64_t e = g.off<double>(x, y, z, S);  // cL; cD, cB, E 128 elements apart
      const double E = fwd64[e + 3 * 128];
      b[0][j] = (T)E;
      if (x < g.nx - 1) b[1][j] = (T)fwd64[g.off<double>(x + 1, y, z, S, 0)];
      if (y < g.ny - 1) b[2][j] = (T)fwd64[g.off<double>(x, y + 1, z, S, 1)];
      if (z < g.nz - 1) b[3][j] = (T)fwd64[g.off<double>(x, y, z + 1, S, 2)];
      if constexpr (sizeof(T) == 4) {
        const double pi = E != 0.0 ? 1.0 / E : 0.0;
        f[0][j] = (T)pi;
        f[1][j] = E != 0.0 ? (T)(2.0 * pi * pi - adiag[g.off<double>(x, y, z)]) : T(0);
        f[2][j] = (T)fwd64[e];
        f[3][j] = (T)fwd64[e + 128];
        f[4][j] = (T)fwd64[e + 256];
        f[5][j] = (T)E;
      }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) chunk_store(o.bwd + c.in_stream<T>(kBwdStream, k), b[k]);
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int k = 0; k < 6; k++) chunk_store(o.fwd + c.in_stream<T>(kFwdStream<T>, k), f[k]);
    }
  }
}
// The matrix in FP32 (the FP32 SpMV of the restarted defect correction).
__global__ void __launch_bounds__(kThreads) k_matrix32(int64_t n, SysArrays<double> a, SysArrays<float> o) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
    o.adiag[e] = (float)a.adiag[e];
    o.al[e] = (float)a.al[e];
    o.ad[e] = (float)a.ad[e];
    o.ab[e] = (float)a.ab[e];
  }
}

// b - A x in FP64 (norms only): the true residual of the final iterate.
__global__ void __launch_bounds__(kThreads)
    k_true_residual(Tiled g, const double* __restrict__ adiag, const double* __restrict__ al,
                    const double* __restrict__ ad, const double* __restrict__ ab,
                    const uint8_t* __restrict__ act, const double* __restrict__ x,
                    const double* __restrict__ b, double* partials, PcgScalars* sc) {
  double s2 = 0.0, mx = 0.0;
  SC_ROWBLOCK_LOOP(g) {
    Cell c;
    c.init(g, rb, threadIdx.x);
    if (c.inside && act[c.e]) {
      const double rv = b[c.e] - apply_row(g, c, adiag, al, ad, ab, act, [&](int dx, int dy, int dz) {
                          return x[dx < 0 ? c.xm(g) : dx > 0 ? c.xp(g) : dy < 0 ? c.ym(g) : dy > 0 ? c.yp(g) : dz < 0 ? c.zm(g) : dz > 0 ? c.zp(g) : c.e];
                        });
      s2 += rv * rv;
      mx = fmax(mx, fabs(rv));
    }
  }
  reduce_finalize(s2, mx, partials, sc, FIN_NORMS);
}

// Mixed precision defect correction: x += scale d ; r -= scale A d (FP64 A, x and r
// in the Tiled layout; the FP32 correction d in the SweepLayout).
__global__ void __launch_bounds__(kThreads)
    k_mixed_update(Tiled g, SweepLayout sg, const double* __restrict__ adiag, const double* __restrict__ al,
                   const double* __restrict__ ad, const double* __restrict__ ab,
                   const uint8_t* __restrict__ act, const float* __restrict__ d, double scale,
                   double* __restrict__ x, double* __restrict__ r, double* partials,
                   PcgScalars* sc) {
  double s2 = 0.0, mx = 0.0;
  SC_ROWBLOCK_LOOP(g) {
    Cell c;
    c.init(g, rb, threadIdx.x);
    if (!(c.inside && act[c.e])) continue;
    const double t = apply_row(g, c, adiag, al, ad, ab, act, [&](int dx, int dy, int dz) {
      return (double)d[sg.off<float>(c.x + dx, c.y + dy, c.z + dz)];
    });
    x[c.e] += scale * (double)d[sg.off<float>(c.x, c.y, c.z)];
    const double rv = r[c.e] - scale * t;
    r[c.e] = rv;
    s2 += rv * rv;
    mx = fmax(mx, fabs(rv));
  }
  reduce_finalize(s2, mx, partials, sc, FIN_NORMS);
}

// SweepArgs::bits of one unit of cx by cy tiles.
template <class Swept>
__host__ __device__ void tile_bits(int2 u, int cx, int cy, Swept swept, uint8_t* out) {
  for (int r = 0; r < cx * cy; r++) {
    const int X = u.x * cx + r % cx, Y = u.y * cy + r / cx;
    out[r] = !swept(X, Y) ? 0
                          : kTileSwept | (swept(X - 1, Y) ? 1 : 0) | (swept(X + 1, Y) ? 2 : 0) | (swept(X, Y - 1) ? 4 : 0) |
                                (swept(X, Y + 1) ? 8 : 0);
  }
}

// The units the iterations visit: the entries of `all` (n of them, in dependency
// order; a unit is cx by cy tiles) that hold an active tile, in the same order, and
// their count in the header entry dst[-1].  Optional: per entry the bits of its tiles
// (SweepArgs::bits), and zeros for the dot-product shares of tiles that are not swept
// (nothing writes those meanwhile).  A block per list.
struct OrderList {
  int cx, cy;
  const int2* all;
  int n;
  int2* dst;
  uint8_t* bits;
  double* tile_partials;
};
struct OrderLists {
  OrderList l[3];
};
__global__ void __launch_bounds__(1024) k_compact_order(int ntx, int nty, const uint8_t* __restrict__ tile_act, OrderLists lists) {
  const OrderList& o = lists.l[blockIdx.x];
  const int cx = o.cx, cy = o.cy, n = o.n;
  const int2* const all = o.all;
  int2* const dst = o.dst;
  uint8_t* const bits = o.bits;
  double* const tile_partials = o.tile_partials;
  __shared__ int wsum[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int b0 = 0; b0 < n; b0 += blockDim.x) {
    const int i = b0 + threadIdx.x;
    bool on = false;
    if (i < n) {
      const int2 u = all[i];
      for (int X = u.x * cx; X < min(ntx, (u.x + 1) * cx); X++)
        for (int Y = u.y * cy; Y < min(nty, (u.y + 1) * cy); Y++) {
          const bool act = tile_act[Y * ntx + X] != 0;
          on |= act;
          if (!act && tile_partials)
            for (int w = 0; w < kSweepWarps; w++) tile_partials[(Y * ntx + X) * kSweepWarps + w] = 0.0;
        }
    }
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (lane == 0) wsum[warp] = __popc(m);
    __syncthreads();
    int before = carry;
    for (int w = 0; w < warp; w++) before += wsum[w];
    before += __popc(m & ((1u << lane) - 1u));
    if (on) {
      dst[before] = all[i];
      if (bits)
        tile_bits(all[i], cx, cy, [&](int X, int Y) { return X >= 0 && X < ntx && Y >= 0 && Y < nty && tile_act[Y * ntx + X]; },
                  bits + (int64_t)before * kMaxCluster);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int t = 0;
      for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += wsum[w];
      carry += t;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) dst[-1] = make_int2(carry, 0);
}

// Writes a header entry (the count) followed by the units of an ntx x nyu
// grid in anti-diagonal order into `o` (ntx nyu + 1 entries).
void all_units_order(int ntx, int nyu, int2* o) {
  int n = 0;
  o[n++] = make_int2(ntx * nyu, 0);
  for (int d = 0; d <= ntx + nyu - 2; d++)
    for (int X = std::max(0, d - nyu + 1); X <= std::min(d, ntx - 1); X++) o[n++] = make_int2(X, d - X);
}
std::vector<int2> all_units_order(int ntx, int nyu) {
  std::vector<int2> o((size_t)ntx * nyu + 1);
  all_units_order(ntx, nyu, o.data());
  return o;
}

// SweepArgs::bits of an order list (header entry first) when every tile is swept.
std::vector<uint8_t> all_tile_bits(const SweepLayout& g, int cx, int cy, const int2* order) {
  std::vector<uint8_t> b((size_t)order[0].x * kMaxCluster, 0);
  for (int i = 0; i < order[0].x; i++)
    tile_bits(order[i + 1], cx, cy, [&](int X, int Y) { return X >= 0 && X < g.ntx && Y >= 0 && Y < g.nty; },
              b.data() + (size_t)i * kMaxCluster);
  return b;
}
// The sweeps of a solver's arrays.
inline PivotOp pivot_op(const PcgSolver::PivotIn& in, double* fwd, double sigma) {
  return {{in.a[0], in.a[1], in.a[2], in.a[3], in.a[4], in.a[5], in.a[6]},
          nullptr,
          {fwd, fwd + 128, fwd + 256, fwd + 384},
          sigma};
}
template <class T, bool SELFDOT = false>
FwdOp<T, SELFDOT> fwd_op(const SysArrays<T>& A) {  // q = L^-1 r
  return {{A.r}, A.fwd + 128 * kFwdFactor<T>, {A.q}};
}
template <class T>
BwdOp<T> bwd_op(const SysArrays<T>& A) {  // z = L^-T q, z.r
  return {{A.q, A.r}, A.bwd, {A.z}};
}

inline int grid_for(int64_t n, int sm) {
  int64_t b = (n + kThreads - 1) / kThreads;
  int64_t cap = (int64_t)sm * 4;
  return (int)std::max<int64_t>(1, std::min(b, cap));
}

}  // namespace

// =================================================================================
// PcgSolver (host)

template <>
cudaGraphExec_t& PcgSolver::graph_for<double>(bool) {
  return graph64_;
}
template <>
cudaGraphExec_t& PcgSolver::graph_for<float>(bool eis) {
  return eis ? graph32e_ : graph32_;
}

void PcgSolver::reset_mailboxes(bool f32) {
  const int64_t qx = sweep_mbx_elems(sg_) * sg_.ntiles() / 4, qy = sweep_mby_elems(sg_) * sg_.ntiles() / 4;
  const int grid = grid_for(std::max(qx, qy), ctx_->sm_count);
  if (f32) {
    k_mb_reset<float><<<grid, kThreads, 0, ctx_->stream>>>(qx, mbx32_);
    k_mb_reset<float><<<grid, kThreads, 0, ctx_->stream>>>(qy, mby32_);
  } else {
    k_mb_reset<double><<<grid, kThreads, 0, ctx_->stream>>>(qx, mbx64_);
    k_mb_reset<double><<<grid, kThreads, 0, ctx_->stream>>>(qy, mby64_);
  }
}

// A sweep of this solver: plan.run<T, FWD>(op, stream).  all_tiles: every tile
// (the pivot sweep), else those with an active cell.
struct PcgSolver::SweepPlan {
  SweepArgs a;
  int clusters;
  template <class T, bool FWD, class Op>
  void run(const Op& op, cudaStream_t st) const {
    launch_sweep<T, FWD>(a, op, st, clusters);
  }
};
PcgSolver::SweepPlan PcgSolver::sweep(bool f32, int use_skip, int fin, bool all_tiles) const {
  SweepPlan p{};
  SweepArgs& w = p.a;
  w.g = sg_;
  w.cx = cl_x_;
  w.cy = cl_y_;
  w.mbx = f32 ? (void*)mbx32_ : (void*)mbx64_;
  w.mby = f32 ? (void*)mby32_ : (void*)mby64_;
  w.ticket = ticket_;
  w.exits = ticket_ + 1;
  w.order = all_tiles ? order_cl_all_ : order_cl_act_;
  w.bits = all_tiles ? bits_all_ : bits_act_;
  w.sc = sc_;
  w.tile_partials = tile_partials_;
  w.col_sums = col_sums_;
  w.t32_sums = t32_sums_;
  w.t32_count = t32_count_;
  w.use_skip = use_skip;
  w.fin_kind = fin;
  p.clusters = cl_grid_;
  return p;
}

int PcgSolver::spin_limit() const { return ctx_->wait_limit > 0 ? ctx_->wait_limit : kSpinLimit; }

int PcgSolver::recover_after_timeout() {
  cudaStream_t st = ctx_->stream;
  reset_mailboxes(false);
  if (have_f32_) reset_mailboxes(true);
  cudaMemsetAsync(sc_, 0, sizeof(PcgScalars), st);
  cudaMemsetAsync(t32_count_, 0, sizeof(int) * (size_t)g_.ntiles(), st);
  pivots_valid_ = false;
  cudaStreamSynchronize(st);
  return ctx_->set_error(-6, "wavefront wait timed out");
}

PcgSolver::PcgSolver(Context* ctx, int nx, int ny, int nz, const PcgOptions& opt)
    : ctx_(ctx), opt_(opt) {
  if (nx < 1 || ny < 1 || nz < 1) {
    init_status_ = -1;
    return;
  }
  g_ = Tiled::make(nx, ny, nz);
  sg_ = SweepLayout::make(nx, ny, nz);
  sweep_set_attr<double, true, PivotOp>();
  sweep_set_attr<double, true, FwdOp<double>>();
  sweep_set_attr<double, false, BwdOp<double>>();
  sweep_set_attr<float, true, FwdOp<float>>();
  sweep_set_attr<float, false, BwdOp<float>>();
  sweep_set_attr<float, true, FwdOp<float, true>>();
  sweep_set_attr<float, false, BwdEisenstatOp<float>>();
  sweep_set_attr<float, true, FwdEisenstatOp<float>>();
  nblocks_ = ctx->sm_count * 8;
  const int ntiles = sg_.ntiles();
  if ((int64_t)sg_.ntx * sg_.nty > kMaxTiles) {
    init_status_ = -3;
    return;
  }
  auto alloc = [&](size_t bytes) -> void* {
    void* p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) return nullptr;
    allocs_.push_back(p);
    return p;
  };
  const size_t nt = sizeof(double) * (size_t)g_.total, ns = sizeof(double) * (size_t)sg_.total;
  double** tiled[] = {&d64_.adiag, &d64_.al, &d64_.ad, &d64_.ab, &rhs_, &press_};
  double** swept[] = {&d64_.r, &d64_.p, &d64_.z, &d64_.s, &d64_.q, &d64_.Az};
  auto alloc_zero = [&](double** a, size_t bytes) {
    *a = (double*)alloc(bytes);
    if (*a) cudaMemsetAsync(*a, 0, bytes, ctx->stream);
    return *a != nullptr;
  };
  bool ok = true;
  for (double** a : tiled) ok = ok && alloc_zero(a, nt);
  for (double** a : swept) ok = ok && alloc_zero(a, ns);
  ok = ok && alloc_zero(&d64_.fwd, ns * kFwdStream<double>) && alloc_zero(&d64_.bwd, ns * kBwdStream);
  if (!ok) {
    init_status_ = -3;
    return;
  }
  active_ = (uint8_t*)alloc((size_t)g_.total);
  partials_ = (double*)alloc(sizeof(double) * 2 * (size_t)nblocks_);
  sc_ = (PcgScalars*)alloc(sizeof(PcgScalars));
  ticket_ = (int*)alloc(sizeof(int) * 2);
  tile_partials_ = (double*)alloc(sizeof(double) * (size_t)ntiles * kSweepWarps);
  tile_act_ = (uint8_t*)alloc((size_t)ntiles);
  // order lists: a header entry (the count) and up to ntiles entries
  col_sums_ = (double*)alloc(sizeof(double) * (size_t)ntiles * kSweepWarps * 32);
  t32_sums_ = (double*)alloc(sizeof(double) * (size_t)g_.ntiles());
  t32_count_ = (int*)alloc(sizeof(int) * (size_t)g_.ntiles());
  int2* order_all = (int2*)alloc(sizeof(int2) * (size_t)(ntiles + 1));
  int2* order = (int2*)alloc(sizeof(int2) * (size_t)(ntiles + 1));
  // mailboxes (FP64; the FP32 ones are allocated with the FP32 arrays)
  mbx64_ = (double*)alloc(sizeof(double) * (size_t)(sweep_mbx_elems(sg_) * ntiles));
  mby64_ = (double*)alloc(sizeof(double) * (size_t)(sweep_mby_elems(sg_) * ntiles));
  if (!active_ || !partials_ || !sc_ || !ticket_ || !order || !order_all || !mbx64_ || !mby64_ ||
      !tile_partials_ || !tile_act_ || !col_sums_ || !t32_sums_ || !t32_count_) {
    init_status_ = -3;
    return;
  }
  order_all_ = order_all + 1;
  order_act_ = order + 1;
  cudaMemsetAsync(ticket_, 0, sizeof(int) * 2, ctx->stream);
  cudaMemsetAsync(t32_count_, 0, sizeof(int) * (size_t)g_.ntiles(), ctx->stream);
  cudaMemsetAsync(active_, 0, (size_t)g_.total, ctx->stream);
  cudaMemsetAsync(sc_, 0, sizeof(PcgScalars), ctx->stream);
  cudaMemsetAsync(partials_, 0, sizeof(double) * 2 * (size_t)nblocks_, ctx->stream);
  reset_mailboxes(false);
  // tile order: anti-diagonals of the tile grid, so every tile's forward
  // predecessors (X-1,Y), (X,Y-1) hold smaller tickets; reversed for backward.
  // Until the first system selects its active tiles, both lists hold all.
  std::vector<int2> ord = all_units_order(sg_.ntx, sg_.nty);
  cudaMemcpyAsync(order_all, ord.data(), sizeof(int2) * ord.size(), cudaMemcpyHostToDevice, ctx->stream);
  cudaMemcpyAsync(order, ord.data(), sizeof(int2) * ord.size(), cudaMemcpyHostToDevice, ctx->stream);
  choose_clusters();
  const int ncx = (sg_.ntx + cl_x_ - 1) / cl_x_, ncy = (sg_.nty + cl_y_ - 1) / cl_y_;
  std::vector<int2> oc = all_units_order(ncx, ncy);
  int2* ca = (int2*)alloc(sizeof(int2) * oc.size());
  int2* cc = (int2*)alloc(sizeof(int2) * oc.size());
  if (!ca || !cc) {
    init_status_ = -3;
    return;
  }
  cudaMemcpyAsync(ca, oc.data(), sizeof(int2) * oc.size(), cudaMemcpyHostToDevice, ctx->stream);
  cudaMemcpyAsync(cc, oc.data(), sizeof(int2) * oc.size(), cudaMemcpyHostToDevice, ctx->stream);
  order_cl_all_ = ca + 1;
  order_cl_act_ = cc + 1;
  const std::vector<uint8_t> bits = all_tile_bits(sg_, cl_x_, cl_y_, oc.data());
  bits_all_ = (uint8_t*)alloc(bits.size());
  bits_act_ = (uint8_t*)alloc(bits.size());
  if (!bits_all_ || !bits_act_) {
    init_status_ = -3;
    return;
  }
  cudaMemcpyAsync(bits_all_, bits.data(), bits.size(), cudaMemcpyHostToDevice, ctx->stream);
  cudaMemcpyAsync(bits_act_, bits.data(), bits.size(), cudaMemcpyHostToDevice, ctx->stream);
  // and the Tiled tiles (two sweep tiles along x), for the SpMV
  std::vector<int2> ot = all_units_order(g_.ntx, g_.nty);
  int2* ta = (int2*)alloc(sizeof(int2) * ot.size());
  int2* tc = (int2*)alloc(sizeof(int2) * ot.size());
  if (!ta || !tc) {
    init_status_ = -3;
    return;
  }
  cudaMemcpyAsync(ta, ot.data(), sizeof(int2) * ot.size(), cudaMemcpyHostToDevice, ctx->stream);
  cudaMemcpyAsync(tc, ot.data(), sizeof(int2) * ot.size(), cudaMemcpyHostToDevice, ctx->stream);
  order_t32_all_ = ta + 1;
  order_t32_act_ = tc + 1;
  if (cudaMallocHost(&sc_host_, sizeof(PcgScalars) * 2) != cudaSuccess) {
    init_status_ = -3;
    return;
  }
  cudaEventCreate(&ev0_);
  cudaEventCreate(&ev1_);
  cudaEventCreate(&evt0_);
  cudaEventCreate(&evt1_);
  if (cudaStreamSynchronize(ctx->stream) != cudaSuccess) init_status_ = -2;
}

// The sweeps' cluster shape.  Inside a cluster boundary values go straight into the
// next block's shared memory, ~0.4 us sooner than through a mailbox.  Where the
// clusters' blocks are no more than the SMs: the shape that leaves the fewest hand-offs
// between clusters (128^3: 2 x 4 clusters of 4 x 4 tiles, FP32 forward sweep 69 us
// against 78 without clusters).  Where tiles have to queue, a cluster holds its SMs
// until its last block is through, and pairs along y are the best of both (256^3
// mixed solve: 127 ms without, 122 with pairs, 130 with 4, 143 with 16).
void PcgSolver::choose_clusters() {
  auto shape = [&](int size, int& cx, int& cy) {  // fewest hand-offs for this size; false if the grid is smaller
    int best = 1 << 30;
    for (int x = 1; x <= size; x *= 2) {
      const int y = size / x;
      if ((x > 1 && x / 2 >= sg_.ntx) || (y > 1 && y / 2 >= sg_.nty)) continue;
      const int n = (sg_.ntx + x - 1) / x + (sg_.nty + y - 1) / y;
      if (n >= best) continue;
      best = n;
      cx = x;
      cy = y;
    }
    return best < (1 << 30);
  };
  int best = 1 << 30;
  for (int size : {1, 2, 4, 8, 16}) {
    int cx, cy;
    if (!shape(size, cx, cy)) continue;
    const int nx = (sg_.ntx + cx - 1) / cx, ny = (sg_.nty + cy - 1) / cy;
    if (nx + ny >= best || (size > 2 && nx * ny * size > ctx_->sm_count)) continue;
    // 16 is beyond the portable size: where the GPU grants it
    if (size > 8 && (sweep_max_clusters<double, true, PivotOp>(size) < 1 ||
                     sweep_max_clusters<float, true, FwdEisenstatOp<float>>(size) < 1))
      continue;
    best = nx + ny;
    cl_x_ = cx;
    cl_y_ = cy;
    cl_grid_ = std::min(nx * ny, ctx_->sm_count / size);
  }
}

PcgSolver::~PcgSolver() {
  if (graph64_) cudaGraphExecDestroy(graph64_);
  if (graph32_) cudaGraphExecDestroy(graph32_);
  if (graph32e_) cudaGraphExecDestroy(graph32e_);
  if (ev0_) cudaEventDestroy(ev0_);
  if (ev1_) cudaEventDestroy(ev1_);
  if (evt0_) cudaEventDestroy(evt0_);
  if (evt1_) cudaEventDestroy(evt1_);
  if (sc_host_) cudaFreeHost(sc_host_);
  for (void* p : allocs_) cudaFree(p);
}

int PcgSolver::check_dev_error(const char* where) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    char buf[256];
    snprintf(buf, sizeof buf, "%s: %s", where, cudaGetErrorString(e));
    return ctx_->set_error(-2, buf);
  }
  return 0;
}

// Staging buffers of the host-array entry points, allocated on first use and
// kept: a per-call stream-ordered allocation can hand its pages back at the
// solve's synchronisations and pay for mapping them again on the next call.
int PcgSolver::ensure_host_stage() {
  if (hstage_) return 0;
  const size_t N = (size_t)g_.nx * g_.ny * g_.nz;
  void *a = nullptr, *b = nullptr;
  if (cudaMalloc(&a, sizeof(double) * N) != cudaSuccess) return ctx_->set_error(-3, "staging allocation failed");
  if (cudaMalloc(&b, N) != cudaSuccess) {
    cudaFree(a);
    return ctx_->set_error(-3, "staging allocation failed");
  }
  allocs_.push_back(a);
  allocs_.push_back(b);
  hstage_ = (double*)a;
  hstage_act_ = (uint8_t*)b;
  return 0;
}

int PcgSolver::upload(const double* adiag, const double* const an[6], const double* rhs,
                      const uint8_t* active, bool device) {
  cudaStream_t st = ctx_->stream;
  const int64_t N = (int64_t)g_.nx * g_.ny * g_.nz;
  const int grid = grid_for(g_.total, ctx_->sm_count);
  const double* src[5] = {adiag, an[0], an[3], an[5], rhs};
  double* dst[5] = {d64_.adiag, d64_.al, d64_.ad, d64_.ab, rhs_};
  // staging buffers for host input (one array at a time)
  double* stage = nullptr;
  uint8_t* stage_act = nullptr;
  if (!device) {
    if (int e = ensure_host_stage()) return e;
    stage = hstage_;
    stage_act = hstage_act_;
    cudaMemcpyAsync(stage_act, active, (size_t)N, cudaMemcpyHostToDevice, st);
  }
  const uint8_t* act_ref = device ? active : stage_act;
  k_to_tiled<uint8_t, uint8_t><<<grid, kThreads, 0, st>>>(g_, act_ref, active_, nullptr);
  launches_ += 6;
  for (int a = 0; a < 5; a++) {
    const double* s = src[a];
    if (!device) {
      cudaMemcpyAsync(stage, src[a], sizeof(double) * (size_t)N, cudaMemcpyHostToDevice, st);
      s = stage;
    }
    // rhs is zeroed outside the active set (the reference never reads it there)
    if (a == 4)
      k_to_tiled<double, double><<<grid, kThreads, 0, st>>>(g_, s, dst[a], act_ref);
    else
      k_matrix_to_tiled<<<grid, kThreads, 0, st>>>(g_, s, dst[a], act_ref, a - 1);
  }
  int rc = 0;
  if (opt_.check_symmetry) {
    const double** dan = nullptr;
    std::vector<double*> tmp;
    double* all = nullptr;
    if (cudaMallocAsync((void**)&dan, sizeof(double*) * 6, st) != cudaSuccess)
      return ctx_->set_error(-3, "upload: allocation failed");
    const double* ptrs[6];
    if (device) {
      for (int d = 0; d < 6; d++) ptrs[d] = an[d];
    } else {
      if (cudaMallocAsync((void**)&all, sizeof(double) * (size_t)N * 6, st) != cudaSuccess)
        return ctx_->set_error(-3, "upload: allocation failed");
      for (int d = 0; d < 6; d++) {
        cudaMemcpyAsync(all + (size_t)N * d, an[d], sizeof(double) * (size_t)N,
                        cudaMemcpyHostToDevice, st);
        ptrs[d] = all + (size_t)N * d;
      }
    }
    cudaMemcpyAsync(dan, ptrs, sizeof(ptrs), cudaMemcpyHostToDevice, st);
    k_symmetry<<<nblocks_, kThreads, 0, st>>>(g_.nx, g_.ny, g_.nz, dan, act_ref, partials_, sc_);
    cudaMemcpyAsync(sc_host_, sc_, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    sym_err_ = sc_host_->rinf;
    cudaFreeAsync(dan, st);
    if (all) cudaFreeAsync(all, st);
    if (sym_err_ > 1e-4) rc = -7;
  }
  pivots_valid_ = false;
  int e = check_dev_error("upload");
  if (e) return e;
  if (rc) return ctx_->set_error(rc, "upload: the matrix is not symmetric (checkSystemSymmetry)");
  return 0;
}

int PcgSolver::upload_rhs(const double* rhs, bool device) {
  cudaStream_t st = ctx_->stream;
  const int64_t N = (int64_t)g_.nx * g_.ny * g_.nz;
  const int grid = grid_for(g_.total, ctx_->sm_count);
  // active_ is already tiled; build a reference-layout mask on the fly is not
  // needed: zero rhs where the tiled mask is 0 after conversion.
  const double* s = rhs;
  double* stage = nullptr;
  if (!device) {
    if (int e = ensure_host_stage()) return e;
    stage = hstage_;
    cudaMemcpyAsync(stage, rhs, sizeof(double) * (size_t)N, cudaMemcpyHostToDevice, st);
    s = stage;
  }
  k_to_tiled<double, double><<<grid, kThreads, 0, st>>>(g_, s, rhs_, nullptr);
  return check_dev_error("upload_rhs");
}

int PcgSolver::download_pressure(double* pg, bool device) {
  cudaStream_t st = ctx_->stream;
  const int64_t N = (int64_t)g_.nx * g_.ny * g_.nz;
  const int grid = grid_for(g_.total, ctx_->sm_count);
  const double* src = press_;
  if (device) {
    k_from_tiled<double, double><<<grid, kThreads, 0, st>>>(g_, src, pg);
    launches_ += 1;
    return check_dev_error("download_pressure");
  }
  if (int e = ensure_host_stage()) return e;
  double* stage = hstage_;
  k_from_tiled<double, double><<<grid, kThreads, 0, st>>>(g_, src, stage);
  launches_ += 1;
  cudaMemcpyAsync(pg, stage, sizeof(double) * (size_t)N, cudaMemcpyDeviceToHost, st);
  if (cudaStreamSynchronize(st) != cudaSuccess) return check_dev_error("download_pressure");
  return check_dev_error("download_pressure");
}

// The matrix in FP32, which only the FP32 SpMV reads (the inner PCG of the mixed solve,
// not the Eisenstat iteration): allocated and made when it is first needed for a system,
// since the inner method may change between two solves of the same one.
int PcgSolver::ensure_matrix32() {
  if (matrix32_valid_) return 0;
  for (float** a : {&d32_.adiag, &d32_.al, &d32_.ad, &d32_.ab}) {
    if (*a) continue;
    void* p = nullptr;
    if (cudaMalloc(&p, sizeof(float) * (size_t)g_.total) != cudaSuccess)
      return ctx_->set_error(-3, "FP32 allocation failed");
    allocs_.push_back(p);
    *a = (float*)p;
  }
  k_matrix32<<<grid_for(g_.total, ctx_->sm_count), kThreads, 0, ctx_->stream>>>(g_.total, d64_, d32_);
  launches_ += 1;
  matrix32_valid_ = true;
  return 0;
}

// The pivots' inputs (PivotOp) in arrays that hold nothing else until the first solve or
// application: the diagonal and the lower couplings in r, p, s and the place of the
// backward factors, the neighbour products in z, q and Az.
PcgSolver::PivotIn PcgSolver::pivot_in() const { return {{d64_.r, d64_.p, d64_.s, d64_.bwd, d64_.z, d64_.q, d64_.Az}}; }

int PcgSolver::ensure_pivots() {
  const bool wants_matrix32 = opt_.precision == PREC_MIXED && opt_.inner_method != INNER_EISENSTAT;
  if (pivots_valid_) return wants_matrix32 ? ensure_matrix32() : 0;
  cudaStream_t st = ctx_->stream;
  const int sgrid = grid_for(sg_.total / 4, ctx_->sm_count);
  // the pivot sweep reports a timeout through the status word: start it clean,
  // with this context's wait bound
  cudaMemsetAsync(&sc_->err, 0, sizeof(unsigned), st);
  pivot_limit_ = spin_limit();
  cudaMemcpyAsync(&sc_->spin_limit, &pivot_limit_, sizeof(int), cudaMemcpyHostToDevice, st);
  // select_active_tiles clears the vectors that hold the pivots' inputs
  const PivotIn in = pivot_in();
  cudaMemsetAsync(tile_act_, 0, (size_t)sg_.ntiles(), st);
  k_sweep_system<<<sgrid, kThreads, 0, st>>>(sg_, g_, d64_.adiag, d64_.al, d64_.ad, d64_.ab, active_, opt_.tau, in, tile_act_);
  sweep(false, 0, FIN_NONE, true).run<double, true>(pivot_op(in, d64_.fwd, opt_.sigma), st);
  k_sweep_factor<double><<<sgrid, kThreads, 0, st>>>(sg_, d64_.fwd, in.a[0], d64_);
  launches_ += 3;
  {
    // the solve's scalars are set over the status word next: read it first
    unsigned* herr = reinterpret_cast<unsigned*>(sc_host_ + 1);
    cudaMemcpyAsync(herr, &sc_->err, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return check_dev_error("pivots");
    if (*herr & DEV_ERR_TIMEOUT) return recover_after_timeout();
  }
  if (opt_.precision == PREC_MIXED) {
    if (!have_f32_) {
      const size_t n32 = sizeof(float) * (size_t)sg_.total;
      float** arr32[] = {&d32_.fwd, &d32_.bwd, &d32_.r, &d32_.p, &d32_.z, &d32_.s, &d32_.q, &d32_.Az};
      for (float** a : arr32) {
        void* p = nullptr;
        const size_t bytes = n32 * (a == &d32_.fwd ? kFwdStream<float> : a == &d32_.bwd ? kBwdStream : 1);
        if (cudaMalloc(&p, bytes) != cudaSuccess) return ctx_->set_error(-3, "FP32 allocation failed");
        allocs_.push_back(p);
        *a = (float*)p;
        cudaMemsetAsync(p, 0, bytes, st);
      }
      void* p = nullptr;
      if (cudaMalloc(&p, sizeof(double) * (size_t)g_.total) != cudaSuccess)
        return ctx_->set_error(-3, "FP64 residual allocation failed");
      allocs_.push_back(p);
      rres_ = (double*)p;
      const int ntiles = sg_.ntiles();
      void *px = nullptr, *py = nullptr;
      if (cudaMalloc(&px, sizeof(float) * (size_t)(sweep_mbx_elems(sg_) * ntiles)) != cudaSuccess ||
          cudaMalloc(&py, sizeof(float) * (size_t)(sweep_mby_elems(sg_) * ntiles)) != cudaSuccess)
        return ctx_->set_error(-3, "FP32 mailbox allocation failed");
      allocs_.push_back(px);
      allocs_.push_back(py);
      mbx32_ = (float*)px;
      mby32_ = (float*)py;
      reset_mailboxes(true);
      have_f32_ = true;
    }
    k_sweep_factor<float><<<sgrid, kThreads, 0, st>>>(sg_, d64_.fwd, in.a[0], d32_);
    launches_ += 1;
  }
  matrix32_valid_ = false;
  if (wants_matrix32)
    if (int e = ensure_matrix32()) return e;
  select_active_tiles();
  int e = check_dev_error("pivots");
  if (e) return e;
  pivots_valid_ = true;
  return 0;
}

// The tiles the iteration sweeps visit: those with an active cell.  A tile left
// out is never written by a sweep, so the vectors the iterations carry start at
// zero everywhere; on a tile without an active cell they then stay zero, as a
// sweep over it would leave them (its pivots and couplings are zero).
void PcgSolver::select_active_tiles() {
  cudaStream_t st = ctx_->stream;
  const int ntiles = sg_.ntiles();
#if !SC_SKIP_EMPTY_TILES
  cudaMemsetAsync(tile_act_, 1, (size_t)ntiles, st);  // every tile swept
#endif
  const int ncx = (sg_.ntx + cl_x_ - 1) / cl_x_, ncy = (sg_.nty + cl_y_ - 1) / cl_y_;
  const OrderLists lists{{{1, 1, order_all_, ntiles, order_act_, nullptr, tile_partials_},
                          {cl_x_, cl_y_, order_cl_all_, ncx * ncy, order_cl_act_, bits_act_, nullptr},
                          {2, 1, order_t32_all_, g_.ntiles(), order_t32_act_, nullptr, nullptr}}};
  k_compact_order<<<3, 1024, 0, st>>>(sg_.ntx, sg_.nty, tile_act_, lists);
  launches_ += 1;
  // columns of tiles that are not swept add zeros
  cudaMemsetAsync(col_sums_, 0, sizeof(double) * (size_t)ntiles * kSweepWarps * 32, st);
  cudaMemsetAsync(t32_sums_, 0, sizeof(double) * (size_t)g_.ntiles(), st);
  const size_t n64 = sizeof(double) * (size_t)sg_.total, n32 = sizeof(float) * (size_t)sg_.total;
  for (double* v : {d64_.r, d64_.p, d64_.z, d64_.s, d64_.q, d64_.Az}) cudaMemsetAsync(v, 0, n64, st);
  if (have_f32_)
    for (float* v : {d32_.r, d32_.p, d32_.z, d32_.s, d32_.q, d32_.Az}) cudaMemsetAsync(v, 0, n32, st);
}

template <class T>
void PcgSolver::launch_spmv(SysArrays<T>& A, cudaStream_t st, int use_skip) {
  // slot runs per tile: about 12 work items per SM (3 resident blocks x 4), runs of
  // at least 16 slots
  const int ntiles = g_.ntiles();
  const int want = 12 * ctx_->sm_count;
  const int runs = std::max(1, std::min((want + ntiles - 1) / ntiles, g_.nz / 16));
  const int grid = std::min(3 * ctx_->sm_count, ntiles * runs);
  k_spmv<T><<<grid, kThreads, 0, st>>>(sg_, g_, order_t32_act_, A.adiag, A.al, A.ad, A.ab, active_, A.s, A.Az, partials_, sc_,
                                       use_skip, runs);
}

template <class T>
void PcgSolver::launch_iteration(SysArrays<T>& A, bool eis) {
  cudaStream_t st = ctx_->stream;
  const bool f32 = sizeof(T) == 4;
  if constexpr (sizeof(T) == 4) {
    if (eis) {
      // CG on L^-1 A L^-T: s = search direction, z = t = L^-T s,
      // Az = w = L^-1 A L^-T s, q = rh (split residual), p = d (FP32 correction).
      // s = rh + beta s ; t = L^-T s ; iteration count and bound
      sweep(true, 1, FIN_SA).template run<T, false>(
          BwdEisenstatOp<T>{{A.q, A.s}, A.bwd, {A.z, A.s}, T(0)}, st);
      sweep(true, 1, FIN_SPMV).template run<T, true>(
          FwdEisenstatOp<T>{{A.s, A.z}, A.fwd, {A.Az}}, st);  // alpha = rho / s.w
      // x += alpha t ; rh -= alpha w ; beta = rho_new / rho
      k_axpy<T><<<nblocks_, kThreads, 0, st>>>(sg_, order_act_, A.z, A.Az, A.p, A.q, partials_, sc_, FIN_EAXPY);
      return;
    }
  }
  launch_spmv<T>(A, st, 1);
  k_axpy<T><<<nblocks_, kThreads, 0, st>>>(sg_, order_act_, A.s, A.Az, A.p, A.r, partials_, sc_);
  sweep(f32, 1, FIN_NONE).template run<T, true>(fwd_op<T>(A), st);
  sweep(f32, 1, FIN_BWD).template run<T, false>(bwd_op<T>(A), st);
  k_sa<T><<<nblocks_, kThreads, 0, st>>>(sg_, order_act_, A.z, A.s, partials_, sc_);
}

// A CUDA graph of `chunk` iterations, captured on first use.  The legacy
// default stream cannot be captured: the graph stays null then and callers
// launch the same kernels directly.
template <class T>
int PcgSolver::ensure_graph(SysArrays<T>& A, bool eis) {
  cudaGraphExec_t& gx = graph_for<T>(eis);
  if (gx) return 0;
  cudaStream_t s = ctx_->stream;
  cudaGraph_t graph = nullptr;
  if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  for (int i = 0; i < opt_.chunk; i++) launch_iteration<T>(A, eis);
  if (cudaStreamEndCapture(s, &graph) != cudaSuccess || !graph) return check_dev_error("end capture");
  if (cudaGraphInstantiate(&gx, graph, 0) != cudaSuccess) {
    cudaGraphDestroy(graph);
    gx = nullptr;
    return check_dev_error("instantiate");
  }
  cudaGraphDestroy(graph);
  return 0;
}

template <class T>
int PcgSolver::run_pcg(SysArrays<T>& A, double tol, int criterion, int max_iter, bool scale_rhs,
                       PcgStats* st, bool eis) {
  cudaStream_t s = ctx_->stream;
  // scalars
  PcgScalars init{};
  init.spin_limit = spin_limit();
  init.tol = tol;
  init.max_iter = max_iter;
  init.criterion = criterion;
  init.done = DONE_RUNNING;
  init.first = 1;
  cudaMemcpyAsync(sc_, &init, sizeof(PcgScalars), cudaMemcpyHostToDevice, s);
  // r = rhs (or the scaled FP64 residual for the mixed inner solve), p = 0
  const double* src = scale_rhs ? rres_ : rhs_;
  const double scale = scale_rhs ? 1.0 / inner_scale_ : 1.0;
  k_init<T><<<nblocks_, kThreads, 0, s>>>(g_, sg_, src, scale, active_, A.r, A.p, partials_, sc_);
  const bool f32 = sizeof(T) == 4;
  eis = eis && f32;
  if (eis) {
    // rh = L^-1 r ; s = rh ; rho = rh.rh
    if constexpr (sizeof(T) == 4)
      sweep(true, 1, FIN_EINIT).template run<T, true>(fwd_op<T, true>(A), s);
    k_copy<T><<<nblocks_, kThreads, 0, s>>>(sg_, order_act_, A.q, A.s, sc_);
  } else {
    // z = M^-1 r ; s = z ; sigma = z.r
    sweep(f32, 1, FIN_NONE).template run<T, true>(fwd_op<T>(A), s);
    sweep(f32, 1, FIN_BWD).template run<T, false>(bwd_op<T>(A), s);
    k_copy<T><<<nblocks_, kThreads, 0, s>>>(sg_, order_act_, A.z, A.s, sc_);
  }
  launches_ += eis ? 3 : 4;
  int e = check_dev_error("pcg init");
  if (e) return e;
  e = ensure_graph<T>(A, eis);
  if (e) return e;
  cudaGraphExec_t gx = graph_for<T>(eis);
  const int per_iter = eis ? 3 : 5;
  // launch chunks, two in flight, until the device reports done
  const int max_chunks = max_iter / std::max(1, opt_.chunk) + 3;
  cudaEvent_t evs[2] = {ev0_, ev1_};
  int launched = 0;
  auto launch_chunk = [&](int c) {
    if (gx)
      cudaGraphLaunch(gx, s);
    else
      for (int i = 0; i < opt_.chunk; i++) launch_iteration<T>(A, eis);
    launches_ += per_iter * (uint64_t)opt_.chunk;
    cudaMemcpyAsync(&sc_host_[c & 1], sc_, sizeof(PcgScalars), cudaMemcpyDeviceToHost, s);
    cudaEventRecord(evs[c & 1], s);
  };
  launch_chunk(launched++);
  if (launched < max_chunks) launch_chunk(launched++);
  for (int c = 0;; c++) {
    if (cudaEventSynchronize(evs[c & 1]) != cudaSuccess) return check_dev_error("pcg chunk");
    if (sc_host_[c & 1].done != DONE_RUNNING) break;
    if (launched >= max_chunks) break;
    launch_chunk(launched++);
  }
  cudaMemcpyAsync(&sc_host_[0], sc_, sizeof(PcgScalars), cudaMemcpyDeviceToHost, s);
  if (cudaStreamSynchronize(s) != cudaSuccess) return check_dev_error("pcg sync");
  last_ = sc_host_[0];
  if (st) {
    st->iterations += last_.iter;
    st->status = last_.done;
    st->residual = last_.res;
    st->device_flags |= last_.err;
  }
  if (last_.err & DEV_ERR_TIMEOUT) return recover_after_timeout();
  return check_dev_error("pcg");
}

int PcgSolver::solve_fp64(PcgStats* st) {
  int e = ensure_pivots();
  if (e) return e;
  e = run_pcg<double>(d64_, opt_.tol, opt_.criterion, opt_.max_iter, false, st);
  // the iterate is handed back whatever came of it: after an error the pressure is that
  // of the failed solve, never an earlier one's
  k_sweep_to_tiled<double><<<grid_for(g_.total, ctx_->sm_count), kThreads, 0, ctx_->stream>>>(sg_, g_, d64_.p, press_);
  launches_ += 1;
  if (e == 0 && (last_.err & DEV_ERR_NONFINITE))
    return ctx_->set_error(-8, "pcg: NaN or Inf in the system or the right-hand side");
  return e ? e : check_dev_error("pcg");
}

// Mixed precision with reliable updates: FP32 CG on the split system
// L^-1 A L^-T (Eisenstat's iteration) that never restarts, with the FP64
// solution and residual carried beside it.  After each graph chunk the host
// reads the recursive split residual ||rh|| / ||rh_0||; once it has dropped by
// reliable_delta since the last update (or predicts convergence), the FP32
// correction d is folded into the FP64 state, x += scale d, r -= scale A d,
// and the split residual is replaced by L^-1 r / scale, keeping the search
// direction (residual replacement in the manner of H. A. van der Vorst and
// Q. Ye, "Residual replacement strategies for Krylov subspace iterative methods
// for the convergence of true residuals", SIAM J. Sci. Comput. 22 (2000)).
// The solve stops when the FP64 residual meets the stopping test.  Replacing
// the residual breaks the identity rh.s = rh.rh that CG's step length relies
// on, so an update that did not lower the FP64 residual, or a recursion whose
// residual grew a hundredfold, restarts the search direction (s = rh).
int PcgSolver::solve_mixed_reliable(PcgStats* st) {
  int e = ensure_pivots();
  if (e) return e;
  cudaStream_t s = ctx_->stream;
  const int grid = grid_for(g_.total, ctx_->sm_count);
  SysArrays<float>& A = d32_;
  // x = 0 ; r = b (FP64)
  k_fill<double><<<grid, kThreads, 0, s>>>(g_.total, press_, 0.0);
  PcgScalars init{};
  init.spin_limit = spin_limit();
  init.tol = 0.0;  // the FP32 recursion never stops itself
  init.max_iter = opt_.max_iter;
  init.criterion = CRIT_REL_L2;
  init.done = DONE_RUNNING;
  cudaMemcpyAsync(sc_, &init, sizeof(PcgScalars), cudaMemcpyHostToDevice, s);
  k_norms<<<nblocks_, kThreads, 0, s>>>(g_.total, rhs_, active_, rres_, partials_, sc_);
  launches_ += 2;
  cudaMemcpyAsync(sc_host_, sc_, sizeof(PcgScalars), cudaMemcpyDeviceToHost, s);
  if (cudaStreamSynchronize(s) != cudaSuccess) return check_dev_error("mixed init");
  if (!std::isfinite(sc_host_->rn2)) return ctx_->set_error(-8, "mixed solve: NaN or Inf in the right-hand side");
  const bool abs_crit = opt_.criterion == CRIT_ABS_LINF;
  const double bnorm = sqrt(sc_host_->rn2);
  double meas = abs_crit ? sc_host_->rinf : (bnorm > 0 ? 1.0 : 0.0);
  int updates = 0, status = DONE_RUNNING, iters = 0, restarts = 0;
  unsigned flags = 0;
  if (meas < opt_.tol) status = DONE_CONVERGED;
  const double scale = bnorm;
  if (status == DONE_RUNNING) {
    // d = 0 ; r32 = r / scale ; rh = L^-1 r32 ; s = rh ; rho = rh.rh
    k_init<float><<<nblocks_, kThreads, 0, s>>>(g_, sg_, rres_, 1.0 / scale, active_, A.r, A.p, partials_, sc_);
    sweep(true, 1, FIN_EINIT).run<float, true>(fwd_op<float, true>(A), s);
    k_copy<float><<<nblocks_, kThreads, 0, s>>>(sg_, order_act_, A.q, A.s, sc_);
    launches_ += 3;
    e = ensure_graph<float>(A, true);
    if (e) return e;
  }
  cudaGraphExec_t gx = graph_for<float>(true);
  cudaEvent_t evs[2] = {ev0_, ev1_};
  auto launch_chunk = [&](int slot) {
    if (gx)
      cudaGraphLaunch(gx, s);
    else
      for (int i = 0; i < opt_.chunk; i++) launch_iteration<float>(A, true);
    launches_ += 3 * (uint64_t)opt_.chunk;
    cudaMemcpyAsync(&sc_host_[slot], sc_, sizeof(PcgScalars), cudaMemcpyDeviceToHost, s);
    cudaEventRecord(evs[slot], s);
  };
  double res_u = 1.0, meas_u = meas;  // split and stopping residuals at the last update
  const int max_chunks = opt_.max_iter / std::max(1, opt_.chunk) + 3;
  int launched = 0, seen = 0;
  while (status == DONE_RUNNING) {
    // keep two chunks in flight; look at the older one
    while (launched - seen < 2 && launched < max_chunks) launch_chunk(launched++ & 1);
    if (seen == launched) {
      status = DONE_MAXITER;
      break;
    }
    if (cudaEventSynchronize(evs[seen & 1]) != cudaSuccess) return check_dev_error("mixed chunk");
    const PcgScalars h = sc_host_[seen & 1];
    seen++;
    const bool dev_stop = h.done != DONE_RUNNING || launched >= max_chunks;
    const double predicted = meas_u * h.res / res_u;
    const bool grew = !(h.res <= 100.0 * res_u);
    if (!(dev_stop || grew || h.res < opt_.reliable_delta * res_u || predicted < 0.5 * opt_.tol)) continue;
    // residual replacement after the chunks in flight
    if (cudaStreamSynchronize(s) != cudaSuccess) return check_dev_error("mixed chunk");
    seen = launched;
    k_mixed_update<<<nblocks_, kThreads, 0, s>>>(g_, sg_, d64_.adiag, d64_.al, d64_.ad, d64_.ab, active_, A.p, scale, press_,
                                                 rres_, partials_, sc_);
    k_init<float><<<nblocks_, kThreads, 0, s>>>(g_, sg_, rres_, 1.0 / scale, active_, A.r, A.p, partials_, sc_,
                                                FIN_NONE);
    sweep(true, 0, FIN_EREPLACE).run<float, true>(fwd_op<float, true>(A), s);
    launches_ += 3;
    cudaMemcpyAsync(&sc_host_[0], sc_, sizeof(PcgScalars), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) return check_dev_error("mixed update");
    const PcgScalars u = sc_host_[0];
    updates++;
    iters = u.iter;
    flags |= u.err;
    const double rel = bnorm > 0 ? sqrt(u.rn2) / bnorm : 0.0;
    meas = abs_crit ? u.rinf : rel;
    if (!std::isfinite(rel)) return ctx_->set_error(-8, "mixed solve: non-finite residual");
    if (u.err & DEV_ERR_TIMEOUT) return recover_after_timeout();
    if (meas < opt_.tol) {
      status = DONE_CONVERGED;
    } else if (u.done == DONE_BREAKDOWN && (!(u.err & DEV_ERR_BREAKDOWN) || (u.err & DEV_ERR_NONFINITE) ||
                                            restarts >= 4 || updates >= opt_.max_outer)) {
      status = DONE_BREAKDOWN;
    } else if (u.done == DONE_BREAKDOWN) {
      // s.w == 0: the FP32 recursion lost its search direction before the FP64
      // residual met the test; restart it from the replaced residual (s = rh)
      const int running = DONE_RUNNING;
      const unsigned keep = u.err & ~(unsigned)DEV_ERR_BREAKDOWN;
      cudaMemcpyAsync(&sc_->done, &running, sizeof(int), cudaMemcpyHostToDevice, s);
      cudaMemcpyAsync(&sc_->err, &keep, sizeof(unsigned), cudaMemcpyHostToDevice, s);
      k_copy<float><<<nblocks_, kThreads, 0, s>>>(sg_, order_act_, A.q, A.s, sc_);
      cudaMemsetAsync(&sc_->beta, 0, sizeof(double), s);
      if (cudaStreamSynchronize(s) != cudaSuccess) return check_dev_error("mixed restart");
      launches_ += 1;
      restarts++;
    } else if (u.done == DONE_MAXITER || launched >= max_chunks || updates >= opt_.max_outer) {
      status = DONE_MAXITER;
    } else if (grew || !(meas < meas_u)) {
      k_copy<float><<<nblocks_, kThreads, 0, s>>>(sg_, order_act_, A.q, A.s, sc_);
      cudaMemsetAsync(&sc_->beta, 0, sizeof(double), s);
      launches_ += 1;
    }
    res_u = u.res;
    meas_u = meas;
  }
  if (st) {
    st->iterations += iters;
    st->outer = updates;
    st->residual = meas;
    st->status = status;
    st->device_flags |= flags;
  }
  return check_dev_error("mixed");
}

int PcgSolver::solve_mixed(PcgStats* st) {
  if (opt_.inner_method == INNER_EISENSTAT) return solve_mixed_reliable(st);
  // Defect correction: FP64 residual and solution, FP32 inner MIC-PCG whose
  // pivots were computed in FP64, restarted after each correction.  Stops on
  // the FP64 residual's stopping test.
  int e = ensure_pivots();
  if (e) return e;
  cudaStream_t s = ctx_->stream;
  const int grid = grid_for(g_.total, ctx_->sm_count);
  // x = 0, r = b
  k_fill<double><<<grid, kThreads, 0, s>>>(g_.total, press_, 0.0);
  launches_ += 2;
  PcgScalars init{};
  init.spin_limit = spin_limit();
  init.tol = 0.0;
  init.max_iter = 1;
  init.criterion = CRIT_REL_L2;
  cudaMemcpyAsync(sc_, &init, sizeof(PcgScalars), cudaMemcpyHostToDevice, s);
  k_norms<<<nblocks_, kThreads, 0, s>>>(g_.total, rhs_, active_, rres_, partials_, sc_);
  cudaMemcpyAsync(sc_host_, sc_, sizeof(PcgScalars), cudaMemcpyDeviceToHost, s);
  if (cudaStreamSynchronize(s) != cudaSuccess) return check_dev_error("mixed init");
  if (!std::isfinite(sc_host_->rn2)) return ctx_->set_error(-8, "mixed solve: NaN or Inf in the right-hand side");
  const double bnorm = sqrt(sc_host_->rn2);
  double rnorm = bnorm;
  double rel = bnorm > 0 ? 1.0 : 0.0;
  int outer = 0;
  const bool abs_crit = opt_.criterion == CRIT_ABS_LINF;
  double meas = abs_crit ? sc_host_->rinf : rel;
  while (meas >= opt_.tol && outer < opt_.max_outer) {
    inner_scale_ = rnorm;
    // the inner solve only needs to reach what is still missing (with margin)
    double want = abs_crit ? opt_.inner_rtol : std::max(opt_.inner_rtol, 0.25 * opt_.tol / rel);
    PcgStats inner{};
    e = run_pcg<float>(d32_, std::min(want, 0.5), CRIT_REL_L2, opt_.max_iter, true, &inner,
                       opt_.inner_method == INNER_EISENSTAT);
    if (e) return e;
    if (st) {
      st->iterations += inner.iterations;
      st->device_flags |= inner.device_flags;
    }
    outer++;
    // x += rnorm d ; r -= rnorm A d   (FP64)
    launches_ += 1;
    k_mixed_update<<<nblocks_, kThreads, 0, s>>>(g_, sg_, d64_.adiag, d64_.al, d64_.ad, d64_.ab, active_, d32_.p, rnorm,
                                                 press_, rres_, partials_, sc_);
    cudaMemcpyAsync(sc_host_, sc_, sizeof(PcgScalars), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) return check_dev_error("mixed update");
    rnorm = sqrt(sc_host_->rn2);
    rel = bnorm > 0 ? rnorm / bnorm : 0.0;
    meas = abs_crit ? sc_host_->rinf : rel;
    if (!std::isfinite(rel)) return ctx_->set_error(-8, "mixed solve: non-finite residual");
    if (inner.status == DONE_BREAKDOWN) break;
  }
  if (st) {
    st->outer = outer;
    st->residual = meas;
    st->status = meas < opt_.tol ? DONE_CONVERGED : DONE_MAXITER;
  }
  return check_dev_error("mixed");
}

int PcgSolver::true_residual(PcgStats* st) {
  cudaStream_t s = ctx_->stream;
  launches_ += 2;
  k_true_residual<<<nblocks_, kThreads, 0, s>>>(g_, d64_.adiag, d64_.al, d64_.ad, d64_.ab, active_, press_, rhs_, partials_, sc_);
  PcgScalars* h = sc_host_ + 1;
  cudaMemcpyAsync(h, sc_, sizeof(PcgScalars), cudaMemcpyDeviceToHost, s);
  // ||b||
  if (cudaStreamSynchronize(s) != cudaSuccess) return check_dev_error("true residual");
  const double rn = sqrt(h->rn2), rinf = h->rinf;
  k_norms<<<nblocks_, kThreads, 0, s>>>(g_.total, rhs_, active_, nullptr, partials_, sc_);
  cudaMemcpyAsync(h, sc_, sizeof(PcgScalars), cudaMemcpyDeviceToHost, s);
  if (cudaStreamSynchronize(s) != cudaSuccess) return check_dev_error("true residual");
  const double bn = sqrt(h->rn2);
  if (st) {
    st->true_rel_l2 = bn > 0 ? rn / bn : 0.0;
    st->true_linf = rinf;
  }
  return check_dev_error("true residual");
}

int PcgSolver::solve(PcgStats* st) {
  PcgStats local{};
  if (!st) st = &local;
  *st = PcgStats{};
  const uint64_t launches0 = launches_;
  cudaEventRecord(evt0_, ctx_->stream);
  int e = opt_.precision == PREC_MIXED ? solve_mixed(st) : solve_fp64(st);
  if (e) return e;
  if (opt_.precision == PREC_MIXED && st->status == DONE_BREAKDOWN && (st->device_flags & DEV_ERR_NONFINITE)) {
    // The FP32 recursion left the FP32 range (a preconditioner with very large
    // eigenvalues: the reference's tau terms at some dt/h) while the system is
    // finite: solve it again with the FP64 iteration.
    PcgStats f{};
    e = solve_fp64(&f);
    if (e) return e;
    st->iterations += f.iterations;
    st->status = f.status;
    st->residual = f.residual;
    st->device_flags |= f.device_flags | DEV_FLAG_FP64_RERUN;
  }
  cudaEventRecord(evt1_, ctx_->stream);
  cudaEventSynchronize(evt1_);
  float ms = 0;
  cudaEventElapsedTime(&ms, evt0_, evt1_);
  st->ms = ms;
  st->sym_err = sym_err_;
  if (opt_.true_residual) {
    e = true_residual(st);
    if (e) return e;
  }
  st->kernel_launches = (int64_t)(launches_ - launches0);
  return 0;
}

int PcgSolver::precond_only(const double* r, double* z) {
  cudaStream_t s = ctx_->stream;
  const int grid = grid_for(sg_.total / 4, ctx_->sm_count);
  int e = ensure_pivots();
  if (e) return e;
  k_ref_to_sweep<double><<<grid, kThreads, 0, s>>>(sg_, r, d64_.r);
  PcgScalars init{};
  init.spin_limit = spin_limit();
  init.done = DONE_RUNNING;
  init.first = 1;
  cudaMemcpyAsync(sc_, &init, sizeof(PcgScalars), cudaMemcpyHostToDevice, s);
  sweep(false, 0, FIN_NONE).run<double, true>(fwd_op<double>(d64_), s);
  sweep(false, 0, FIN_BWD).run<double, false>(
      bwd_op<double>(d64_), s);
  k_sweep_to_ref<double><<<grid, kThreads, 0, s>>>(sg_, d64_.z, z);
  cudaMemcpyAsync(sc_host_, sc_, sizeof(PcgScalars), cudaMemcpyDeviceToHost, s);
  if (cudaStreamSynchronize(s) != cudaSuccess) return check_dev_error("precond");
  last_ = *sc_host_;
  if (sc_host_->err & DEV_ERR_TIMEOUT) return recover_after_timeout();
  return check_dev_error("precond");
}

int PcgSolver::apply_only(const double* x, double* b) {
  cudaStream_t s = ctx_->stream;
  const int grid = grid_for(g_.total, ctx_->sm_count);
  // A row reads its neighbours' x while other blocks write b, so overlapping x and b go
  // through a copy, in an array whose values no call keeps (and whose padding is zero).
  const size_t bytes = sizeof(double) * (size_t)g_.nx * g_.ny * g_.nz;
  const uintptr_t xa = (uintptr_t)x, ba = (uintptr_t)b;
  const bool overlap = xa < ba + bytes && ba < xa + bytes;
  if (overlap) {
    cudaMemcpyAsync(d64_.Az, x, bytes, cudaMemcpyDeviceToDevice, s);
    x = d64_.Az;
  }
  k_apply_checked<<<grid, kThreads, 0, s>>>(g_, d64_.adiag, d64_.al, d64_.ad, d64_.ab, active_, x, b);
  if (overlap) cudaMemsetAsync(d64_.Az, 0, bytes, s);
  if (cudaStreamSynchronize(s) != cudaSuccess) return check_dev_error("apply");
  return check_dev_error("apply");
}


int PcgSolver::time_kernels(int reps, double* ms) {
  cudaStream_t s = ctx_->stream;
  int e = ensure_pivots();
  if (e) return e;
  const int grid = grid_for(g_.total, ctx_->sm_count);
  // a benign state: r = rhs, s = r, scalars running with a tiny alpha/beta
  PcgScalars init{};
  init.spin_limit = spin_limit();
  init.done = DONE_RUNNING;
  init.first = 1;
  init.max_iter = 1 << 30;
  init.alpha = 0.0;
  init.beta = 0.0;
  init.sigma = 1.0;
  // The mixed solver iterates in FP32: time its FP32 kernels (the pivot sweep
  // is FP64 in both).
  const bool f32 = opt_.precision == PREC_MIXED && have_f32_;
  auto kernel = [&](auto& A, int which) {
    using T = std::remove_reference_t<decltype(*A.r)>;
    const SweepPlan plan = sweep(sizeof(T) == 4, 0, FIN_NONE);
    switch (which) {
      case 1:
        plan.template run<T, true>(fwd_op<T>(A), s);
        break;
      case 2:
        plan.template run<T, false>(bwd_op<T>(A), s);
        break;
      case 3:
        launch_spmv<T>(A, s, 0);
        break;
      case 4:
        k_axpy<T><<<nblocks_, kThreads, 0, s>>>(sg_, order_act_, A.s, A.Az, A.p, A.r, partials_, sc_);
        break;
      case 5:
        k_sa<T><<<nblocks_, kThreads, 0, s>>>(sg_, order_act_, A.z, A.s, partials_, sc_);
        break;
      case 6:
        if constexpr (sizeof(T) == 4)
          plan.template run<T, false>(BwdEisenstatOp<T>{{A.q, A.s}, A.bwd, {A.z, A.s}, T(0)}, s);
        break;
      case 7:
        if constexpr (sizeof(T) == 4)
          plan.template run<T, true>(FwdEisenstatOp<T>{{A.s, A.z}, A.fwd, {A.Az}}, s);
        break;
    }
  };
  auto benign_state = [&]() -> int {
    cudaMemcpyAsync(sc_, &init, sizeof(PcgScalars), cudaMemcpyHostToDevice, s);
    k_init<double><<<nblocks_, kThreads, 0, s>>>(g_, sg_, rhs_, 1.0, active_, d64_.r, d64_.p, partials_, sc_);
    cudaMemcpyAsync(sc_, &init, sizeof(PcgScalars), cudaMemcpyHostToDevice, s);
    k_copy<double><<<grid, kThreads, 0, s>>>(sg_, order_act_, d64_.r, d64_.s, sc_);
    if (f32) {
      if ((e = ensure_matrix32())) return e;
      k_init<float><<<nblocks_, kThreads, 0, s>>>(g_, sg_, rhs_, 1.0, active_, d32_.r, d32_.p, partials_, sc_);
      cudaMemcpyAsync(sc_, &init, sizeof(PcgScalars), cudaMemcpyHostToDevice, s);
      k_copy<float><<<grid, kThreads, 0, s>>>(sg_, order_act_, d32_.r, d32_.s, sc_);
    }
    return 0;
  };
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  auto timed = [&](int which) -> double {
    cudaEventRecord(a, s);
    for (int i = 0; i < reps; i++) {
      switch (which) {
        case 0: {
          // the pivots' inputs live in the solve's arrays only until that starts; rebuild them
          const PivotIn in = pivot_in();
          k_sweep_system<<<grid, kThreads, 0, s>>>(sg_, g_, d64_.adiag, d64_.al, d64_.ad, d64_.ab, active_, opt_.tau, in, nullptr);
          sweep(false, 0, FIN_NONE, true).run<double, true>(pivot_op(in, d64_.fwd, opt_.sigma), s);
          k_sweep_factor<double><<<grid, kThreads, 0, s>>>(sg_, d64_.fwd, in.a[0], d64_);
          break;
        }
        default:
          if (f32)
            kernel(d32_, which);
          else
            kernel(d64_, which);
          break;
      }
    }
    cudaEventRecord(b, s);
    cudaEventSynchronize(b);
    float t = 0;
    cudaEventElapsedTime(&t, a, b);
    return (double)t / reps;
  };
  for (int k = 0; k < 8 && !e; k++) {
    cudaMemcpyAsync(sc_, &init, sizeof(PcgScalars), cudaMemcpyHostToDevice, s);
    ms[k] = (k < 6 || f32) ? timed(k) : 0.0;
    if (k == 0) e = benign_state();
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  return e ? e : check_dev_error("time_kernels");
}

}  // namespace sc

// =================================================================================
// Allocation-free MIC(0) preconditioner (sc_mic_precond_noalloc_device).
//
// Some callers cannot call cudaMalloc: engines whose device memory is owned up
// front by their own pool allocator (no third-party allocations allowed), and
// hot loops where cudaMalloc's implicit device-wide synchronisation is not
// acceptable.  For them this variant of ModifiedIncompleteCholesky3D::precond
// keeps every scratch buffer it needs (the tiled copies of A, the pivots, the
// sweep couplings, the sweep outputs, the tile mailboxes and the scheduling
// counters) in the file-scope array below instead of allocating.  It launches
// the same kernels as sc_pcg_precond_device.
//
// The array is kNoAllocBytes (about 8.5 MB) and lives on every GPU that loads
// this library, until the process exits.  It bounds the problem size: at most
// kNoAllocMaxTiled tiled elements (ceil(nx/32)*32 * ceil(ny/8)*8 * nz, e.g. a
// 32^3 grid) in at most kNoAllocMaxTiles column tiles.  Every call shares the
// one array, so calls whose work overlaps on the GPU (other streams, other
// host threads) race and corrupt each other's results.
namespace sc {
namespace {

constexpr int64_t kNoAllocMaxTiled = 32768;
constexpr int kNoAllocMaxTiles = 8;
constexpr int kNoAllocTiledArrays = 4;   // adiag al ad ab
constexpr int kNoAllocSweptArrays = 16;  // adiag al ad ab, fwd (4), bwd (4), r q z Az

// chunks of a warp tile of the tallest grid of `tiles` column tiles, and the
// largest SweepLayout among the grids accepted (the padding weighs most at 8
// tiles of 16 cells)
constexpr int na_chunks(int tiles) { return (int)(kNoAllocMaxTiled / (tiles * 256) + 10 + 3) / 4; }  // Tiled tiles, two sweep tiles each
constexpr int64_t na_max_swept() {
  int64_t m = 0;
  for (int t = 1; t <= kNoAllocMaxTiles; t++) m = (int64_t)t * na_chunks(t) * 1024 > m ? (int64_t)t * na_chunks(t) * 1024 : m;
  return m;
}
constexpr size_t na_align(size_t b) { return (b + 255) & ~(size_t)255; }
constexpr size_t kNaTiledBytes = na_align(sizeof(double) * kNoAllocMaxTiled);
constexpr size_t kNaSweptBytes = na_align(sizeof(double) * na_max_swept());
constexpr size_t kNaActBytes = na_align(kNoAllocMaxTiled);
// mailboxes: 32 and 64 values per sweep tile and chunk, 512 cells per tile and chunk
constexpr size_t kNaMbxBytes = na_align(sizeof(double) * na_max_swept() / 16);
constexpr size_t kNaMbyBytes = na_align(sizeof(double) * na_max_swept() / 8);
constexpr int kNaSweepTiles = 2 * kNoAllocMaxTiles;
constexpr size_t kNaSmallBytes = na_align(sizeof(double) * kNaSweepTiles * kSweepWarps + sizeof(int) * 2 +
                                          sizeof(int2) * (kNaSweepTiles + 1) + kNaSweepTiles * kMaxCluster) +
                                 na_align(sizeof(PcgScalars));
constexpr size_t kNoAllocBytes = kNaTiledBytes * kNoAllocTiledArrays + kNaSweptBytes * kNoAllocSweptArrays +
                                 kNaActBytes + kNaMbxBytes + kNaMbyBytes + kNaSmallBytes;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

std::mutex g_noalloc_mutex;
void* g_noalloc_base[64] = {};  // device address of g_noalloc_scratch, per device

}  // namespace

// Returns 0, or a negative status with `msg` set.
int mic_precond_noalloc(cudaStream_t st, int device, int sm_count, int nx, int ny, int nz,
                        const double* adiag, const double* const* an, const double* r,
                        const uint8_t* active, double* z, double tau, double sigma,
                        std::string* msg) {
  const Tiled g = Tiled::make(nx, ny, nz);
  if (g.total > kNoAllocMaxTiled || g.ntiles() > kNoAllocMaxTiles) {
    *msg = "grid too large for the allocation-free preconditioner: at most " +
           std::to_string(kNoAllocMaxTiled) + " tiled cells (ceil(nx/32)*32 * ceil(ny/8)*8 * nz) in " +
           std::to_string(kNoAllocMaxTiles) + " tiles of 32x8 columns";
    return -1;
  }
  if (device < 0 || device >= 64) {
    *msg = "device ordinal out of range";
    return -1;
  }
  unsigned char* base = nullptr;
  {
    // One-time set-up per device (the device is current here): the device
    // address of the static array, and the shared-memory attribute of the sweeps.
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_base[device]) {
      void* ptr = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
      if (e != cudaSuccess || !ptr) {
        *msg = std::string("cudaGetSymbolAddress failed: ") + cudaGetErrorString(e);
        return -2;
      }
      sweep_set_attr<double, true, PivotOp>();
      sweep_set_attr<double, true, FwdOp<double>>();
      sweep_set_attr<double, false, BwdOp<double>>();
      g_noalloc_base[device] = ptr;
    }
    base = (unsigned char*)g_noalloc_base[device];
  }
  const SweepLayout sg = SweepLayout::make(nx, ny, nz);
  unsigned char* q = base;
  auto take = [&q](size_t bytes) {
    unsigned char* p = q;
    q += bytes;
    return p;
  };
  double* tl[kNoAllocTiledArrays];
  for (double*& a : tl) a = (double*)take(kNaTiledBytes);
  double* arr[kNoAllocSweptArrays];
  for (double*& a : arr) a = (double*)take(kNaSweptBytes);
  uint8_t* act = (uint8_t*)take(kNaActBytes);
  double* mbx = (double*)take(kNaMbxBytes);
  double* mby = (double*)take(kNaMbyBytes);
  double* tile_partials = (double*)q;
  int* ticket = (int*)(tile_partials + kNaSweepTiles * kSweepWarps);
  int2* order = (int2*)(ticket + 2);  // header entry, then the tiles
  uint8_t* bits = (uint8_t*)(order + kNaSweepTiles + 1);
  PcgScalars* scal = (PcgScalars*)(q + kNaSmallBytes - na_align(sizeof(PcgScalars)));
  SysArrays<double> A;
  A.r = arr[12], A.q = arr[13], A.z = arr[14], A.Az = arr[15];
  A.fwd = arr[4], A.bwd = arr[8];  // four arrays each
  // The array keeps the previous call's contents: reset what must start at
  // zero (scheduling counters, scalars) and the mailbox sentinels.
  const int ntiles = sg.ntiles();
  const int64_t mqx = sweep_mbx_elems(sg) * ntiles / 4, mqy = sweep_mby_elems(sg) * ntiles / 4;
  // An error left pending by earlier, unrelated work is not this call's.
  cudaGetLastError();
  auto failed = [&](cudaError_t e, const char* step) {
    if (e == cudaSuccess) return false;
    *msg = std::string(step) + ": " + cudaGetErrorString(e);
    return true;
  };
  if (failed(cudaMemsetAsync(ticket, 0, sizeof(int) * 2, st), "clearing the tile tickets") ||
      failed(cudaMemsetAsync(scal, 0, sizeof(PcgScalars), st), "clearing the status word"))
    return -2;
  const int rgrid = grid_for(mqy, sm_count);
  k_mb_reset<double><<<rgrid, kThreads, 0, st>>>(mqx, mbx);
  k_mb_reset<double><<<rgrid, kThreads, 0, st>>>(mqy, mby);
  if (failed(cudaGetLastError(), "resetting the mailboxes")) return -2;
  // every tile is swept (the order of all tiles, its count in the header)
  int2 ord[kNaSweepTiles + 1];
  all_units_order(sg.ntx, sg.nty, ord);
  if (failed(cudaMemcpyAsync(order, ord, sizeof(int2) * (ntiles + 1), cudaMemcpyHostToDevice, st),
             "uploading the tile order"))
    return -2;
  const std::vector<uint8_t> hbits = all_tile_bits(sg, 1, 1, ord);
  if (failed(cudaMemcpyAsync(bits, hbits.data(), hbits.size(), cudaMemcpyHostToDevice, st), "uploading the tile bits"))
    return -2;
  // system into the tiled layout and from there into the sweeps'; right-hand side
  const int grid = grid_for(g.total, sm_count);
  k_to_tiled<uint8_t, uint8_t><<<grid, kThreads, 0, st>>>(g, active, act, nullptr);
  k_matrix_to_tiled<<<grid, kThreads, 0, st>>>(g, adiag, tl[0], active, -1);
  k_matrix_to_tiled<<<grid, kThreads, 0, st>>>(g, an[0], tl[1], active, 0);
  k_matrix_to_tiled<<<grid, kThreads, 0, st>>>(g, an[3], tl[2], active, 1);
  k_matrix_to_tiled<<<grid, kThreads, 0, st>>>(g, an[5], tl[3], active, 2);
  const int sgrid = grid_for(sg.total / 4, sm_count);
  const PcgSolver::PivotIn in{{arr[0], arr[1], arr[2], arr[3], A.z, A.q, A.Az}};
  k_sweep_system<<<sgrid, kThreads, 0, st>>>(sg, g, tl[0], tl[1], tl[2], tl[3], act, tau, in, nullptr);
  k_ref_to_sweep<double><<<sgrid, kThreads, 0, st>>>(sg, r, A.r);
  if (failed(cudaGetLastError(), "converting the system to the solver's layouts")) return -2;
  // pivots, couplings, forward and backward sweeps
  SweepArgs wa{};
  wa.g = sg;
  wa.cx = wa.cy = 1;
  wa.mbx = mbx;
  wa.mby = mby;
  wa.ticket = ticket;
  wa.exits = ticket + 1;
  wa.order = order + 1;
  wa.bits = bits;
  wa.sc = scal;
  wa.tile_partials = tile_partials;
  wa.col_sums = nullptr;  // no dot product is wanted
  wa.use_skip = 0;
  wa.fin_kind = FIN_NONE;
  const int wgrid = std::min(ntiles, 2 * sm_count);
  launch_sweep<double, true>(wa, pivot_op(in, A.fwd, sigma), st, wgrid);
  k_sweep_factor<double><<<sgrid, kThreads, 0, st>>>(sg, A.fwd, in.a[0], A);
  launch_sweep<double, true>(wa, fwd_op<double>(A), st, wgrid);
  launch_sweep<double, false>(wa, bwd_op<double>(A), st, wgrid);
  k_sweep_to_ref<double><<<sgrid, kThreads, 0, st>>>(sg, A.z, z);
  if (failed(cudaGetLastError(), "launching the pivot and sweep kernels")) return -2;
  unsigned err = 0;
  if (failed(cudaMemcpyAsync(&err, &scal->err, sizeof(unsigned), cudaMemcpyDeviceToHost, st),
             "reading the status word") ||
      failed(cudaStreamSynchronize(st), "running the preconditioner") ||
      failed(cudaGetLastError(), "running the preconditioner"))
    return -2;
  if (err & DEV_ERR_TIMEOUT) {
    *msg = "wavefront wait timed out";
    return -6;
  }
  return 0;
}

}  // namespace sc
