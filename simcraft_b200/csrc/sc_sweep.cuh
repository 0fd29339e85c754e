// sc_sweep.cuh -- the wavefront sweeps of the MIC(0) preconditioner on B200.
//
// A sweep evaluates a recurrence in which a cell needs the values of its three
// lower (forward) or upper (backward) neighbours: ModifiedIncompleteCholesky3D::precond
// (FluidSim/src/cpu/project-solver.cc:230-306), its pivots, and the two sweeps of
// the Eisenstat iteration.  The i+j+k order leaves 3n - 2 dependent steps, so a
// sweep is bound by the time of one step and of a hand-off between the units
// that own neighbouring columns, until the grid is large enough for HBM.
//
// Units.  A warp owns 8 x 4 columns (SweepLayout).  Inside it the x and y
// neighbours arrive by shuffle and the z neighbour is the lane's previous value:
// a step has no memory access and no barrier in its dependent chain.  Warps hand
// their boundary values on every four steps (a chunk), through rings in shared
// memory within a block, and through mailboxes in global memory between blocks;
// in both a word that holds no value holds a sentinel.  A value is then its own flag,
// and so is its absence: a warp stores a value only into words in which it has read
// the sentinel, so the accesses to each word order one another and no fence or barrier
// is involved.  (An mbarrier per ring entry cost ~400 cycles of a chunk's ~1100;
// divergent branches around the hand-off another ~400.  Separate words in which a
// consumer says how far it is need a fence before them, and a fence waits for the
// stores of the outputs: 256^3 mixed solve 175 ms.  The look at the words instead is
// asked for three chunks before its answer is needed, in rings long enough for that:
// 127 ms; with the answer awaited in the same chunk, from rings of half the length,
// 136, and the FP32 sweeps of 512^3 took 908 and 956 us instead of 728 and 766.)
// A block of 4 such warps sweeps a 16 x 8 column tile.
// Four steps per hand-off: the lag it adds (a chunk per warp crossed) costs less
// than a wait per step would, and it is the largest number for which both
// boundary offsets (8 and 4 columns) fall on whole chunks.
//
// Streams.  Each lane keeps its own vectors of the next chunks of the sweep's
// input arrays in flight as 16-byte asynchronous copies into its own words of
// shared memory (no other lane reads them, so they need no barrier), across the
// end of a tile into the next one it is going to sweep.
//
// Tiles are handed out by ticket in dependency order (a tile's predecessors hold
// smaller tickets, so the smallest unfinished ticket can always run: no
// co-residency is needed), and a block fetches the next ticket while it is
// finishing its tile.  Every wait is bounded: on timeout the kernel raises
// DEV_ERR_TIMEOUT, stops waiting and finishes.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>
#include <utility>

#include "sc_common.cuh"
#include "sc_pcg.cuh"

namespace sc {
namespace {

__device__ void finalize(int kind, PcgScalars* sc, double sum, double mx);

constexpr int kSpinLimit = 1 << 22;  // default bound of the waits: seconds, far above any legitimate wait

// Cell operations of the sweeps.  Each reads at its own cell NX vectors and NF
// consecutive arrays of a stream of FS (fac points at the first of them), in that
// order in v, plus the three already-computed neighbour values xn, yn, zn; writes
// NO arrays (o; arrays of a stream of OS); and returns the value the recurrence
// passes on to the neighbours.
//
// The factor streams: forward cL, cD, cB, E, in FP32 with Pinv, Dt before them;
// backward E, uR, uU, uF.
template <class T>
constexpr int kFwdStream = sizeof(T) == 4 ? 6 : 4;
template <class T>
constexpr int kFwdFactor = sizeof(T) == 4 ? 2 : 0;  // index of cL
constexpr int kBwdStream = 4;

template <class T, bool SELFDOT = false>
struct FwdOp {  // L q = r (project-solver.cc:276-288), c* = A_* E(neighbour); SELFDOT: acc q.q
  static constexpr int NX = 1, NF = 4, FS = kFwdStream<T>, NO = 1, OS = 1;
  const T* src[NX];  // r
  const T* fac;      // cL, cD, cB, E
  T* out[NO];        // q
  __device__ __forceinline__ T step(const T* v, T xn, T yn, T zn, T* o, double& acc) const {
    T t = v[0];
    t -= v[1] * xn;
    t -= v[2] * yn;
    t -= v[3] * zn;
    const T q = t * v[4];
    o[0] = q;
    if (SELFDOT) acc += (double)q * (double)q;
    return q;
  }
};

template <class T>
struct BwdOp {  // L^T z = q (project-solver.cc:293-305), u* = A_*(p+dir) E(p); sigma = z.r
  static constexpr int NX = 2, NF = 4, FS = kBwdStream, NO = 1, OS = 1;
  const T* src[NX];  // q, r
  const T* fac;      // E, uR, uU, uF
  T* out[NO];        // z
  __device__ __forceinline__ T step(const T* v, T xn, T yn, T zn, T* o, double& acc) const {
    T t = v[0];
    t -= v[3] * xn;
    t -= v[4] * yn;
    t -= v[5] * zn;
    T z = t * v[2];
    o[0] = z;
    acc += (double)z * (double)v[1];
    return z;
  }
};

// Eisenstat backward sweep with the search-direction update folded in:
//   s = rh + beta s  (scaleAndAdd of the CG step), then t = L^-T s.
// beta comes from the device scalars, read once per block (prepare).
template <class T>
struct BwdEisenstatOp {
  static constexpr int NX = 2, NF = 4, FS = kBwdStream, NO = 2, OS = 1;
  const T* src[NX];  // rh, s (previous)
  const T* fac;      // E, uR, uU, uF
  T* out[NO];        // t, s (in place of src[1]: each element is read before it is written)
  T beta;
  __device__ __forceinline__ void prepare(const PcgScalars* sc) { beta = (T)sc->beta; }
  __device__ __forceinline__ T step(const T* v, T xn, T yn, T zn, T* o, double&) const {
    const T sv = v[0] + beta * v[1];
    o[1] = sv;
    T u = sv;
    u -= v[3] * xn;
    u -= v[4] * yn;
    u -= v[5] * zn;
    const T t = u * v[2];
    o[0] = t;
    return t;
  }
};

// Ops without per-launch scalars.
template <class Op, class = void>
struct HasPrepare : std::false_type {};
template <class Op>
struct HasPrepare<Op, std::void_t<decltype(std::declval<Op&>().prepare(nullptr))>> : std::true_type {};

// Eisenstat's form of the preconditioned operator (S. C. Eisenstat, "Efficient
// implementation of a class of preconditioned conjugate gradient methods",
// SIAM J. Sci. Stat. Comput. 2 (1981) 1-4).  With the MIC(0) factor
// L = (P^-2 + F) P (P = diag(E), F the strictly lower part of A) and
// A = K + K^T - Dt, K = P^-2 + F, Dt = 2 P^-2 - diag(A), the split operator is
//   L^-1 A L^-T v = P^-1 t + L^-1 (P^-1 v - Dt t),   t = L^-T v,
// so one backward sweep (t) and this forward sweep apply it: no SpMV.  The
// recurrence carries q = L^-1 (P^-1 v - Dt t); the output is w = P^-1 t + q
// and acc gathers v.w.  Pinv = 1/E and Dt are 0 on cells where E = 0.
template <class T>
struct FwdEisenstatOp {
  static constexpr int NX = 2, NF = 6, FS = kFwdStream<T>, NO = 1, OS = 1;
  const T* src[NX];  // v, t
  const T* fac;      // Pinv, Dt, cL, cD, cB, E
  T* out[NO];        // w
  __device__ __forceinline__ T step(const T* v, T xn, T yn, T zn, T* o, double& acc) const {
    T u = v[2] * v[0];
    u -= v[3] * v[1];
    u -= v[4] * xn;
    u -= v[5] * yn;
    u -= v[6] * zn;
    const T q = u * v[7];
    const T w = v[2] * v[1] + q;
    o[0] = w;
    acc += (double)v[0] * (double)w;
    return q;
  }
};

// MIC(0) pivot (project-solver.cc:237-274), FP64.  The exchanged value is E.
// E(q) != 0 exactly when q is active with Adiag(q) != 0, which is the guard the
// reference tests before using E(q).  adm is Adiag masked by the active flag;
// dL/dD/dB hold the tau-weighted products with the diagonal neighbours'
// couplings (k_sweep_system), so the sweep only streams its own column.
// A step is three divisions, a square root and another division one after another.
// Only inactive cells branch around them; a term that is absent divides 1 by 1, since
// 0 / x leaves the fast path of the division for the whole warp.  A 16 x 8 x 8192 column
// tile 1007 -> 546 ns a step; 32^3 150 -> 94 us, 128^3 688 -> 583 us, 256^3 2420 -> 1900
// us, half of the cells fluid, with k_sweep_system and k_sweep_factor.  (Without the
// branch for inactive cells 118, 701 and 2340 us.)
struct PivotOp {
  static constexpr int NX = 7, NF = 0, FS = 1, NO = 4, OS = kFwdStream<double>;
  const double* src[NX];  // adm, al, ad, ab, dL, dD, dB
  const double* fac;
  double* out[NO];        // cL, cD, cB, E
  double sigma;
  __device__ __forceinline__ double step(const double* v, double EL, double ED, double EB, double* o, double&) const {
    const double adiag = v[0], al = v[1], ad = v[2], ab = v[3];
    double E = 0.0;
    if (adiag != 0.0) {
      const bool qL = EL != 0.0 && v[4] != 0.0, qD = ED != 0.0 && v[5] != 0.0, qB = EB != 0.0 && v[6] != 0.0;
      const double tL = (qL ? v[4] : 1.0) / (qL ? EL * EL : 1.0), tD = (qD ? v[5] : 1.0) / (qD ? ED * ED : 1.0),
                   tB = (qB ? v[6] : 1.0) / (qB ? EB * EB : 1.0);
      double ee = adiag;
      ee -= (al * EL) * (al * EL);
      ee = qL ? ee - tL : ee;
      ee -= (ad * ED) * (ad * ED);
      ee = qD ? ee - tD : ee;
      ee -= (ab * EB) * (ab * EB);
      ee = qB ? ee - tB : ee;
      if (ee < sigma * adiag) ee = adiag;
      E = 1.0 / sqrt(ee);
    }
    o[0] = al * EL;
    o[1] = ad * ED;
    o[2] = ab * EB;
    o[3] = E;
    return E;
  }
};

// Arguments of one sweep launch.
struct SweepArgs {
  SweepLayout g;
  int cx, cy;             // tiles of a cluster along x and y
  void *mbx, *mby;        // mailboxes of each consumer tile: [nc][8 rows][4], [nc][16 columns][4]
  int *ticket, *exits;    // next ticket; blocks that found no more tiles
  const int2* order;      // cluster tiles (x, y) in dependency order, their count in order[-1].x
  // per entry of order and rank of the cluster: kTileSwept if the rank's tile is swept,
  // and 1, 2, 4, 8 if the tile at X - 1, X + 1, Y - 1, Y + 1 of it is.  A tile without an
  // active cell is not: it holds zeros and has zero couplings to its neighbours.
  const uint8_t* bits;
  PcgScalars* sc;
  double* tile_partials;  // per tile and warp: the warp's share of an FP32 sweep's dot product
  // FP64 sweeps: per column (tile, warp, lane) its share, per 32 x 8 columns their sum,
  // and the warps of those that are done (null col_sums: no dot product)
  double *col_sums, *t32_sums;
  int* t32_count;
  int use_skip;
  int fin_kind;
};
constexpr int kMaxCluster = 16;  // blocks of a cluster (the stride of SweepArgs::bits)
constexpr int kTileSwept = 16;

// A block's ticket word: the number of its tile (Y * ntx + X) and the tile's bits above
// it; kNoTile: no more tiles.  A grid has at most kMaxTiles tiles, so that their columns
// have 32-bit numbers (a tile takes over 200 KB of a solver's arrays: these are
// exhausted long before).
constexpr int kTileBits = 27;
constexpr int kMaxTiles = (1 << 24) - 1;
constexpr unsigned kNoTile = 0xffffffffu;
// the word of block `rank` of a cluster at `unit`
__host__ __device__ __forceinline__ unsigned ticket_pack(const SweepLayout& g, int cx, int cy, int2 unit, int rank, unsigned bits) {
  const int X = unit.x * cx + rank % cx, Y = unit.y * cy + rank / cx;
  return (bits ? (unsigned)(Y * g.ntx + X) : 0u) | bits << kTileBits;  // a tile that is not swept may lie outside the grid
}
__host__ __device__ __forceinline__ int ticket_tile(unsigned w) { return (int)(w & ((1u << kTileBits) - 1)); }
__host__ __device__ __forceinline__ int ticket_bits(unsigned w) { return (int)(w >> kTileBits); }
inline int64_t sweep_mbx_elems(const SweepLayout& g) { return (int64_t)g.nc * SweepLayout::TY * 4; }  // per tile
inline int64_t sweep_mby_elems(const SweepLayout& g) { return (int64_t)g.nc * SweepLayout::TX * 4; }

// ---- primitives -----------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// Shared memory of another block of the cluster: the address there of what is at p here.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t p, int rank) {
  uint32_t q;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(q) : "r"(p), "r"(rank));
  return q;
}
__device__ __forceinline__ int cluster_rank() {
  int r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.aligned;\n barrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ int ld_shared(uint32_t p) {
  int v;
  asm volatile("ld.volatile.shared.s32 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_shared64(uint32_t p) {
  unsigned long long v;
  asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(v) : "r"(p) : "memory");
  return v;
}
// stores to cluster addresses
__device__ __forceinline__ void st_cluster64(uint32_t p, unsigned long long v) {
  asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void add_cluster(uint32_t p, int v) {
  asm volatile("red.relaxed.cluster.shared::cluster.add.s32 [%0], %1;" ::"r"(p), "r"(v) : "memory");
}
// 16-byte copy global -> shared past L1, visible to this thread after cp_async_wait.
// Off, nothing is written either: copies in flight to one place are not ordered, so a
// zero fill of a slot could land on the data that is copied there next.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p cp.async.cg.shared.global [%0], [%1], 16;\n}\n" ::"r"(dst),
               "l"(src), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Hand-off words (mailboxes and rings).  Every access is a strong operation, and
// an empty word holds the sentinel, a NaN payload that arithmetic never produces:
// a consumer that reads anything else has the value; it then writes the sentinel
// back, which makes the word free for its producer's next value: that is stored only
// where the sentinel has been read (a mailbox entry takes one value in a launch).
template <class T>
struct Sentinel;
template <>
struct Sentinel<double> {
  using Bits = unsigned long long;
  static constexpr Bits bits = 0x7ff4deadbeefcafeull;
};
template <>
struct Sentinel<float> {
  using Bits = unsigned int;
  static constexpr Bits bits = 0x7fa5deadu;
};
template <class T>
struct Quad {  // four values of one lane
  T e[4];
};
__device__ __forceinline__ Quad<float> mb_load(const float* p) {
  Quad<float> q;
  asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(q.e[0]), "=f"(q.e[1]), "=f"(q.e[2]), "=f"(q.e[3])
               : "l"(p)
               : "memory");
  return q;
}
__device__ __forceinline__ Quad<double> mb_load(const double* p) {
  Quad<double> q;
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(q.e[0]), "=d"(q.e[1]) : "l"(p) : "memory");
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(q.e[2]), "=d"(q.e[3]) : "l"(p + 2) : "memory");
  return q;
}
// The stores are predicated, not branched around: a divergent branch costs tens of
// cycles of a chunk's few hundred.
__device__ __forceinline__ void mb_store(float* p, const Quad<float>& q, bool on = true) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.s32 p, %5, 0;\n @p st.relaxed.gpu.global.v4.f32 [%0], {%1, %2, %3, %4};\n}\n" ::"l"(p),
      "f"(q.e[0]), "f"(q.e[1]), "f"(q.e[2]), "f"(q.e[3]), "r"((int)on)
      : "memory");
}
__device__ __forceinline__ void mb_store(double* p, const Quad<double>& q, bool on = true) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.s32 p, %5, 0;\n @p st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};\n"
      " @p st.relaxed.gpu.global.v2.f64 [%0+16], {%3, %4};\n}\n" ::"l"(p),
      "d"(q.e[0]), "d"(q.e[1]), "d"(q.e[2]), "d"(q.e[3]), "r"((int)on)
      : "memory");
}
template <class T>
__device__ __forceinline__ Quad<T> sentinel_quad() {
  Quad<T> q;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    if constexpr (sizeof(T) == 8)
      q.e[i] = __longlong_as_double((long long)Sentinel<T>::bits);
    else
      q.e[i] = __uint_as_float(Sentinel<T>::bits);
  }
  return q;
}
template <class T>
__device__ __forceinline__ bool is_sentinel(T v) {
  if constexpr (sizeof(T) == 8)
    return __double2hiint(v) == (int)(Sentinel<T>::bits >> 32);  // no other value has this high word
  else
    return __float_as_uint(v) == Sentinel<T>::bits;
}
template <class T>
__device__ __forceinline__ bool mb_full(const Quad<T>& q) {
  return !(is_sentinel(q.e[0]) | is_sentinel(q.e[1]) | is_sentinel(q.e[2]) | is_sentinel(q.e[3]));
}
// A sum that is NaN if any of the words is the sentinel (and seldom otherwise: a
// true NaN, or double values whose high words overflow a float): one addition
// tree and one comparison where mb_full needs four.
__device__ __forceinline__ float sentinel_probe(const Quad<float>& q) { return (q.e[0] + q.e[1]) + (q.e[2] + q.e[3]); }
__device__ __forceinline__ float sentinel_probe(const Quad<double>& q) {
  return (__int_as_float(__double2hiint(q.e[0])) + __int_as_float(__double2hiint(q.e[1]))) +
         (__int_as_float(__double2hiint(q.e[2])) + __int_as_float(__double2hiint(q.e[3])));
}
template <class T>
__device__ __forceinline__ bool mb_empty(const Quad<T>& q) {
  return is_sentinel(q.e[0]) & is_sentinel(q.e[1]) & is_sentinel(q.e[2]) & is_sentinel(q.e[3]);
}

// A lane's four values of a chunk at element p (SweepLayout::within).
__device__ __forceinline__ Quad<float> chunk_load(const float* p) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  return {{a.x, a.y, a.z, a.w}};
}
__device__ __forceinline__ Quad<double> chunk_load(const double* p) {
  const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 64);
  return {{a.x, a.y, b.x, b.y}};
}
__device__ __forceinline__ void chunk_store(float* p, const float* v) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void chunk_store(double* p, const double* v) {
  *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
  *reinterpret_cast<double2*>(p + 64) = make_double2(v[2], v[3]);
}
// A ring entry of one lane: four consecutive values at shared-memory address p.
template <class T>
__device__ __forceinline__ Quad<T> ring_load(uint32_t p) {
  Quad<T> q;
  if constexpr (sizeof(T) == 4) {
    asm volatile("ld.volatile.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(q.e[0]), "=f"(q.e[1]), "=f"(q.e[2]), "=f"(q.e[3])
                 : "r"(p)
                 : "memory");
  } else {
    asm volatile("ld.volatile.shared.v2.f64 {%0, %1}, [%2];" : "=d"(q.e[0]), "=d"(q.e[1]) : "r"(p) : "memory");
    asm volatile("ld.volatile.shared.v2.f64 {%0, %1}, [%2];" : "=d"(q.e[2]), "=d"(q.e[3]) : "r"(p + 16) : "memory");
  }
  return q;
}
__device__ __forceinline__ void ring_store(uint32_t p, const Quad<float>& q, bool on = true) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.s32 p, %5, 0;\n @p st.volatile.shared.v4.f32 [%0], {%1, %2, %3, %4};\n}\n" ::"r"(p),
      "f"(q.e[0]), "f"(q.e[1]), "f"(q.e[2]), "f"(q.e[3]), "r"((int)on)
      : "memory");
}
__device__ __forceinline__ void ring_store(uint32_t p, const Quad<double>& q, bool on = true) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.s32 p, %5, 0;\n @p st.volatile.shared.v2.f64 [%0], {%1, %2};\n"
      " @p st.volatile.shared.v2.f64 [%0+16], {%3, %4};\n}\n" ::"r"(p),
      "d"(q.e[0]), "d"(q.e[1]), "d"(q.e[2]), "d"(q.e[3]), "r"((int)on)
      : "memory");
}

// The same into a ring of a block of the cluster (cluster address).
__device__ __forceinline__ void ring_give(uint32_t p, const Quad<float>& q, bool on) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.s32 p, %5, 0;\n @p st.relaxed.cluster.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};\n}\n" ::"r"(p),
      "f"(q.e[0]), "f"(q.e[1]), "f"(q.e[2]), "f"(q.e[3]), "r"((int)on)
      : "memory");
}
__device__ __forceinline__ void ring_give(uint32_t p, const Quad<double>& q, bool on) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.s32 p, %5, 0;\n @p st.relaxed.cluster.shared::cluster.v2.f64 [%0], {%1, %2};\n"
      " @p st.relaxed.cluster.shared::cluster.v2.f64 [%0+16], {%3, %4};\n}\n" ::"r"(p),
      "d"(q.e[0]), "d"(q.e[1]), "d"(q.e[2]), "d"(q.e[3]), "r"((int)on)
      : "memory");
}

// The words of a ring entry of a block of the cluster, and whether any holds a value
// (not zero).
struct RingWords {
  uint32_t w[4];  // FP64: the high words
  __device__ __forceinline__ uint32_t held(uint32_t sentinel) const {
    return (w[0] ^ sentinel) | (w[1] ^ sentinel) | (w[2] ^ sentinel) | (w[3] ^ sentinel);
  }
};
template <class T>
__device__ __forceinline__ RingWords ring_look(uint32_t p) {
  RingWords r;
  if constexpr (sizeof(T) == 4) {
    asm volatile("ld.relaxed.cluster.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3])
                 : "r"(p)
                 : "memory");
  } else {
    unsigned long long q[4];
    asm volatile("ld.relaxed.cluster.shared::cluster.v2.u64 {%0, %1}, [%2];" : "=l"(q[0]), "=l"(q[1]) : "r"(p) : "memory");
    asm volatile("ld.relaxed.cluster.shared::cluster.v2.u64 {%0, %1}, [%2];" : "=l"(q[2]), "=l"(q[3]) : "r"(p + 16) : "memory");
#pragma unroll
    for (int i = 0; i < 4; i++) r.w[i] = (uint32_t)(q[i] >> 32);
  }
  return r;
}

// ---- shared memory of a sweep block -----------------------------------------------
constexpr int kSweepWarps = SweepLayout::kWarps;       // compute warps, 2 (x) by 2 (y)
constexpr int kSweepThreads = (kSweepWarps + 4) * 32;  // + 2 x and 2 y mailbox loaders
constexpr int kRing = 16;                              // entries of a boundary ring: four groups
constexpr int kTick = 8;                               // tickets a block can hold
template <class T, int NV>
struct SweepSmem {
  static constexpr int chunk = 128 * (int)sizeof(T);  // bytes of a chunk of one array
  // chunks staged per warp: 8, or 4 where those do not fit
  static constexpr int ring_bytes = kSweepWarps * kRing * 12 * 4 * (int)sizeof(T);
  static constexpr int room = 227 * 1024;
  static constexpr int D = (room - ring_bytes - 2048) / (kSweepWarps * NV * chunk) >= 8 ? 8 : 4;
  static constexpr int stage = 0;                                     // [warp][D][NV][chunk]
  static constexpr int ringx = stage + kSweepWarps * D * NV * chunk;  // [warp][entry][4 rows][4]
  static constexpr int ringy = ringx + kSweepWarps * kRing * 16 * (int)sizeof(T);  // [warp][entry][8 columns][4]
  static constexpr int tick = ringy + kSweepWarps * kRing * 32 * (int)sizeof(T);  // u64 [kTick]
  static constexpr int acks = tick + kTick * 8;   // int [kTick]
  static constexpr int misc = acks + kTick * 4;  // abort flag, last flag
  static constexpr int sums = misc + 16;
  static constexpr int bytes = sums + kSweepThreads / 32 * 8;
  static_assert(bytes <= room, "a sweep block's shared memory");
};

// What a compute warp copies while it sweeps group gi of a tile's NC chunks (groups of
// four): the first `chunks` chunks of group `group` of this tile or the next one, DG
// groups further on, into the slots that the group's own chunks leave.  ahead: groups of
// the next tile already being copied; has_next: that tile is known and is swept.
// One group of copies is committed per chunk, the empty ones too, and each chunk waits
// for all but the last 4 * DG - 1, so a slot's last copy has landed before the next one
// into it is issued.
struct SweepAhead {
  bool next;
  int group, chunks;
};
__host__ __device__ __forceinline__ SweepAhead sweep_ahead(int gi, int NC, int DG, int ahead, bool has_next) {
  const int NG = (NC + 3) >> 2, g = gi + DG;
  const bool next = g >= NG;
  const int group = next ? g - NG : g;
  const bool on = group < NG && (!next || (has_next && ahead == group));
  const int left = NC - 4 * group;
  return {next, group, on ? (left < 4 ? left : 4) : 0};
}

struct SweepWait {
  PcgScalars* sc;
  uint32_t abort;  // shared-memory word: another wait of this block gave up
  int limit;
  __device__ __forceinline__ bool aborted() const {
    int v;
    asm volatile("ld.volatile.shared.s32 %0, [%1];" : "=r"(v) : "r"(abort) : "memory");
    return v != 0;
  }
  __device__ __forceinline__ void set_abort() const {
    asm volatile("st.volatile.shared.s32 [%0], 1;" ::"r"(abort) : "memory");
  }
  // true: keep waiting
  __device__ __forceinline__ bool more(int& spins, int lim) const {
    ++spins;
    if ((spins & 15) == 0 && aborted()) return false;
    // another block's wait gave up
    if ((spins & 63) == 0 && (ld_relaxed_gpu_u32(&sc->err) & DEV_ERR_TIMEOUT)) {
      set_abort();
      return false;
    }
    if (spins > lim) {
      atomicOr(&sc->err, DEV_ERR_TIMEOUT);
      set_abort();
      return false;
    }
    return true;
  }
};

// Feeds the boundary ring of one compute warp whose producer is in another block:
// moves each mailbox entry on as it fills, q = first .. nq - 1, ring entry e0 + q.
// LPE lanes hold an entry, and every lane moves its own words on by itself; the
// warp polls 32 / LPE entries at once.
template <class T, int LPE>
__device__ void sweep_loader(const SweepWait& W, T* mb, int stride, int first, int nq, uint32_t ring, unsigned e0) {
  constexpr int EP = 32 / LPE, kVec = 4 * (int)sizeof(T);
  const int lane = threadIdx.x & 31, r = lane % LPE;
  int q = first + lane / LPE, spins = 0;
  while (__any_sync(kFull, q < nq)) {
    bool moved = false;
    if (q < nq) {
      T* p = mb + (int64_t)q * stride + r * 4;
      const uint32_t slot = ring + ((e0 + q) % kRing * LPE + r) * kVec;
      const Quad<T> v = mb_load(p), old = ring_load<T>(slot);
      if (mb_full(v) && mb_empty(old)) {
        ring_store(slot, v);
        mb_store(p, sentinel_quad<T>());
        q += EP;
        moved = true;
      }
    }
    if (__any_sync(kFull, moved)) {
      spins = 0;
    } else {
      if (!__all_sync(kFull, W.more(spins, W.limit))) return;
      __nanosleep(16);
    }
  }
}

template <class T, bool FWD, class Op>
__global__ void __launch_bounds__(kSweepThreads, 1)
    k_sweep(const __grid_constant__ SweepArgs a, const __grid_constant__ Op op_arg) {
  constexpr int NX = Op::NX, NF = Op::NF, NV = NX + NF, NO = Op::NO;
  using SM = SweepSmem<T, NV>;
  constexpr int D = SM::D;
  constexpr int kLane = 16 / (int)sizeof(T);  // elements of a lane's vector
  extern __shared__ __align__(1024) unsigned char dyn[];
  // the scalars of the launch in one round trip
  const int running = a.sc->done, spin_limit = a.sc->spin_limit, nticket = a.order[-1].x;
  const unsigned err0 = ld_relaxed_gpu_u32(&a.sc->err);
  if (a.use_skip && running != DONE_RUNNING) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const SweepLayout& g = a.g;
  const int NC = g.nc;
  int* s_misc = reinterpret_cast<int*>(dyn + SM::misc);  // abort flag, last flag
  constexpr int kVec = 4 * (int)sizeof(T);  // bytes of a lane's ring entry
  const uint32_t ringx = smem_u32(dyn + SM::ringx), ringy = smem_u32(dyn + SM::ringy), s_tick = smem_u32(dyn + SM::tick),
                 s_acks = smem_u32(dyn + SM::acks);
  const int rank = cluster_rank(), nrank = a.cx * a.cy, rkx = rank % a.cx, rky = rank / a.cx;
  const int leader = FWD ? 0 : nrank - 1;  // the block whose first warp draws the cluster's tickets
  for (int i = threadIdx.x; i < kSweepWarps * kRing * 12; i += blockDim.x) ring_store(ringx + i * kVec, sentinel_quad<T>());
  for (int i = threadIdx.x; i < (SM::sums - SM::tick) / 4; i += blockDim.x) reinterpret_cast<int*>(dyn + SM::tick)[i] = 0;
  __syncthreads();
  // an earlier sweep gave up: sweep nothing
  if (threadIdx.x == 0) s_misc[0] = (err0 & DEV_ERR_TIMEOUT) ? 1 : 0;
  cluster_sync();
  const SweepWait W{a.sc, smem_u32(s_misc), spin_limit > 0 ? spin_limit : kSpinLimit};
  const int lim = W.limit > (1 << 28) ? (1 << 30) : 4 * W.limit;  // waits behind the mailbox loaders' own bound
  // (in shared memory the ticket's running number + 1 stands above the word)
  auto ticket_word = [&](int t) -> unsigned {  // lane r: the word of rank r
    if (t >= nticket || lane >= nrank) return kNoTile;
    const int at = FWD ? t : nticket - 1 - t;
    const int2 e = a.order[at];
    return ticket_pack(g, a.cx, a.cy, e, lane, a.bits[(int64_t)at * kMaxCluster + lane]);
  };
  // gives ticket n to the cluster's blocks, once all their warps have read the one
  // that held its place (one warp of the leader; a warp counts itself when the word it
  // read has come back, so a later store cannot change what it read)
  auto publish = [&](int n, unsigned w) {
    const int need = n / kTick * (nrank * (kSweepThreads / 32));
    int spins = 0;
    while (!__all_sync(kFull, ld_shared(s_acks + n % kTick * 4) >= need))
      if (!__all_sync(kFull, W.more(spins, lim))) break;
    if (lane < nrank) st_cluster64(cluster_addr(s_tick + n % kTick * 8, lane), (unsigned long long)(n + 1) << 32 | w);
    __syncwarp();
  };
  // the word of ticket n if it is out
  auto peek = [&](int n, unsigned& w) -> bool {
    const unsigned long long v = ld_shared64(s_tick + n % kTick * 8);
    w = (unsigned)v;
    return __all_sync(kFull, (unsigned)(v >> 32) == (unsigned)(n + 1)) != 0;
  };
  auto acquire = [&](int n) -> unsigned {
    unsigned w = kNoTile;
    int spins = 0;
    bool ok = !__any_sync(kFull, W.aborted());
    while (ok && !peek(n, w)) {
      ok = __all_sync(kFull, W.more(spins, lim));
      __nanosleep(n ? 40 : 0);
    }
    if (lane == 0) add_cluster(cluster_addr(s_acks + n % kTick * 4, leader), 1);
    return ok ? w : kNoTile;
  };
  struct Tile {
    int id, nb;
  };
  // this block's tile: false if it is not swept
  auto tile_of = [&](unsigned w, Tile& t) -> bool {
    t.id = ticket_tile(w);
    t.nb = ticket_bits(w);
    return t.nb & kTileSwept;
  };
  const int first = FWD ? 0 : kSweepWarps - 1;  // the compute warp that starts a tile's wave
  // the neighbouring blocks' tiles that are in the same cluster: producers and consumers
  const bool cin_x = FWD ? rkx > 0 : rkx < a.cx - 1, cin_y = FWD ? rky > 0 : rky < a.cy - 1;
  const bool cout_x = FWD ? rkx < a.cx - 1 : rkx > 0, cout_y = FWD ? rky < a.cy - 1 : rky > 0;

  if (warp >= kSweepWarps) {
    // mailbox loaders: warps 4, 5 the x boundary of the two warp rows, 6, 7 the y
    // boundary of the two warp columns
    const int l = (warp - kSweepWarps) & 1;
    const bool isx = warp < kSweepWarps + 2;
    const int cw = isx ? l * 2 + (FWD ? 0 : 1) : (FWD ? 0 : 2) + l;
    unsigned e0 = 0;
    for (int n = 0;; n++, e0 += (NC + 3) & ~3) {
      const unsigned w = acquire(n);
      if (w == kNoTile) break;
      Tile tl;
      if (!tile_of(w, tl)) continue;
      const int tid = tl.id;
      if (isx) {
        if ((tl.nb & (FWD ? 1 : 2)) && !cin_x)  // entry 0 is not needed
          sweep_loader<T, 4>(W, (T*)a.mbx + (int64_t)tid * NC * 32 + l * 16, 32, 1, NC, ringx + cw * kRing * 4 * kVec, e0);
      } else if ((tl.nb & (FWD ? 4 : 8)) && !cin_y) {
        sweep_loader<T, 8>(W, (T*)a.mby + (int64_t)tid * NC * 64 + l * 32, 64, 0, NC, ringy + cw * kRing * 8 * kVec, e0);
      }
    }
  } else {
    Op op = op_arg;
    if constexpr (HasPrepare<Op>::value) op.prepare(a.sc);
    const int cw = warp, wx = cw & 1, wy = cw >> 1, tx = lane & 7, ty = lane >> 3;
    const bool inner_x = FWD ? wx == 0 : wx == 1, inner_y = FWD ? wy == 0 : wy == 1;  // the consumer is in this block
    const bool xedge = FWD ? tx == 0 : tx == 7, yedge = FWD ? ty == 0 : ty == 3;      // lanes fed from outside the warp
    const bool xlast = FWD ? tx == 7 : tx == 0, ylast = FWD ? ty == 3 : ty == 0;      // lanes feeding the next warp
    const int nwx = cw ^ 1, nwy = cw ^ 2;  // the warps that consume (or, in a block before this one, produce) across x and y
    // this lane's words in the rings it reads (row ty, column tx) and feeds
    const uint32_t rx = ringx + (cw * kRing * 4 + ty) * kVec, ry = ringy + (cw * kRing * 8 + tx) * kVec;
    const int dx = FWD ? 1 : -1, dy = FWD ? a.cx : -a.cx;  // rank of the next block along x and y, from this one's
    const uint32_t orx = cluster_addr(ringx + (nwx * kRing * 4 + ty) * kVec, inner_x || !cout_x ? rank : rank + dx),
                   ory = cluster_addr(ringy + (nwy * kRing * 8 + tx) * kVec, inner_y || !cout_y ? rank : rank + dy);
    constexpr uint32_t kSlotX = 4 * kVec, kSlotY = 8 * kVec;
    const T* stage = reinterpret_cast<const T*>(dyn + SM::stage) + cw * D * NV * 128 + lane * kLane;
    const uint32_t stage_u32 = smem_u32(stage);
    // copies this lane's vectors of a chunk (at element v of a vector, f of the factor
    // stream) into stage slot `slot`; off: no chunk
    auto copy = [&](int64_t v, int64_t f, int slot, bool on) {
#pragma unroll
      for (int k = 0; k < NV; k++) {
        const T* p = k < NX ? op.src[k < NX ? k : 0] + v : op.fac + (f + (k - NX) * 128);
        cp_async16(stage_u32 + (slot * NV + k) * SM::chunk, p, on);
        if constexpr (sizeof(T) == 8) cp_async16(stage_u32 + (slot * NV + k) * SM::chunk + 512, p + 64, on);
      }
    };
    constexpr int DG = D / 4;  // groups of four chunks in flight
    // the next ticket is drawn, looked up and published after three successive groups
    // of four chunks, so that nothing waits for its latency
    const int NG = (NC + 3) >> 2, pub_at = NG - 4 - DG;
    const bool publisher = rank == leader && cw == first;
    int next_ticket = 0, pub = 3;
    unsigned next_word = kNoTile;
    auto advance_ticket = [&](int n) {
      if (pub == 0 && lane == 0) next_ticket = atomicAdd(a.ticket, 1);
      if (pub == 1) next_word = ticket_word(__shfl_sync(kFull, next_ticket, 0));
      if (pub == 2) publish(n + 1, W.aborted() ? kNoTile : next_word);
      pub++;
      __syncwarp();
    };
    if (publisher) {
      for (pub = 0; pub < 3;) advance_ticket(-1);
    }
    int ahead = 0;  // groups of the next tile already being copied
    int group = 0;  // running number of groups of four chunks; ring entries 4 * group ...
    // The words of four entries there, which the lanes look at together: 4 x 4 rows, 4 x 8
    // columns.  held: some of the next group's held a value then, or nobody looked.
    const bool rings_x = inner_x || cout_x, rings_y = inner_y || cout_y;
    const uint32_t look_x = orx + (lane >> 3) * kSlotX + ((lane & 3) - ty) * kVec,
                   look_y = ory + (lane >> 3) * kSlotY + ((lane & 7) - tx) * kVec;
    constexpr uint32_t kEmpty = sizeof(T) == 8 ? (uint32_t)((unsigned long long)Sentinel<T>::bits >> 32) : (uint32_t)Sentinel<T>::bits;
    bool held = true;
    for (int n = 0;; n++) {
      const unsigned tw = acquire(n);
      if (tw == kNoTile) break;
      Tile tl;
      pub = 0;
      if (!tile_of(tw, tl)) {
        if (publisher)
          while (pub < 3) advance_ticket(n);
        group += NG;
        held = true;
        ahead = 0;
        continue;
      }
      const int nb = tl.nb, tid = tl.id;
      const int64_t c0 = ((int64_t)tid * kSweepWarps + cw) * NC;
      auto chunk_at = [&](int64_t first_chunk, int d) { return first_chunk + (FWD ? d : NC - 1 - d); };
      // the first groups, as far as they are not on their way
      const bool late = ahead < min(DG, NG);
      if (late) {
        for (; ahead < min(DG, NG); ahead++)
          for (int i = 0; i < 4; i++) {
            const bool in = 4 * ahead + i < NC;
            const int64_t c = chunk_at(c0, in ? 4 * ahead + i : 0);
            copy(c * 128 + lane * kLane, c * (Op::FS * 128) + lane * kLane, (4 * (group + ahead) + i) & (D - 1), in);
            if (n == 0) cp_async_commit();  // a group per chunk, as later
          }
        if (n == 0) {
          for (int i = 4 * min(DG, NG); i < D; i++) cp_async_commit();
        } else {
          cp_async_commit();
          cp_async_wait<0>();
        }
      }
      ahead = 0;
      bool next_known = false;
      int64_t nc0 = -1;  // first chunk of the next tile (-1: none)
      const bool has_x = !inner_x || (nb & (FWD ? 1 : 2)), has_y = !inner_y || (nb & (FWD ? 4 : 8));
      // the consumers of this warp's boundary values: a warp of the cluster or a mailbox
      const bool next_x = nb & (FWD ? 2 : 1), next_y = nb & (FWD ? 8 : 4);
      const bool feeds_x = inner_x || (next_x && cout_x), feeds_y = inner_y || (next_y && cout_y);
      const bool out_x = next_x && !feeds_x, out_y = next_y && !feeds_y;
      T* mox = (T*)a.mbx + (int64_t)(FWD ? tid + 1 : tid - 1) * NC * 32 + (wy * 4 + ty) * 4;
      T* moy = (T*)a.mby + (int64_t)(FWD ? tid + g.ntx : tid - g.ntx) * NC * 64 + (wx * 8 + tx) * 4;
      // Lanes that take a neighbour's value from a ring.  Without a neighbour (a domain
      // edge, or a tile without an active cell) the coupling is zero and what the
      // shuffle brings from another row of the warp serves as well as anything.
      const bool from_x = xedge && has_x, from_y = yedge && has_y;
      // waits for the ring entries at px and py, as far as wanted, and frees their words
      auto take = [&](bool want_x, uint32_t px, bool want_y, uint32_t py, Quad<T>& xq, Quad<T>& yq, auto between) {
        xq = ring_load<T>(px);
        yq = ring_load<T>(py);
        between();
        auto ready = [&] {
          const float gx = sentinel_probe(xq), gy = sentinel_probe(yq);
          const float probe = (want_x ? gx : 0.0f) + (want_y ? gy : 0.0f);
          return __all_sync(kFull, probe == probe) != 0;
        };
        int spins = 0;
        while (!ready()) {
          if ((++spins & 15) == 0) {
            // a true NaN among the values, or a wait that goes on
            if (__all_sync(kFull, (!want_x | mb_full(xq)) & (!want_y | mb_full(yq)))) break;
            int s = spins >> 4;
            if (!__all_sync(kFull, W.more(s, lim))) break;
          }
          xq = ring_load<T>(px);
          yq = ring_load<T>(py);
        }
        ring_store(px, sentinel_quad<T>(), want_x & xedge);
        ring_store(py, sentinel_quad<T>(), want_y & yedge);
      };
      double acc = 0.0;
      T prev = T(0);
      // ring entries of the current group
      uint32_t cur = (group * 4) % kRing;
      // the last value of the entries before the first chunk's: x entry 1, y entry 0
      Quad<T> x0, y0;
      take(has_x, rx + (cur + 1) * kSlotX, has_y, ry + cur * kSlotY, x0, y0, [] {});
      T xc = x0.e[3], yc = y0.e[3];
      // four chunks from d0 on; main part: none of what they take from the rings has ended
      auto four_chunks = [&](auto main_part, int d0) {
        constexpr bool kMain = decltype(main_part)::value;
        const uint32_t nxt = (cur + 4) % kRing;
        const uint32_t rxa = rx + cur * kSlotX, rxb = rx + nxt * kSlotX, rya = ry + cur * kSlotY, ryb = ry + nxt * kSlotY,
                       oxa = orx + cur * kSlotX, oya = ory + cur * kSlotY;
        const int sbase = D == 8 ? (int)(cur & 4) : 0;  // stage slots sbase .. sbase + 3, then the others
        constexpr int kDir = FWD ? 1 : -1;
        const int64_t cg = chunk_at(c0, d0);
        const int64_t ato = cg * (Op::OS * 128) + lane * kLane;
        T* bx = mox + (int64_t)d0 * 32;
        T* by = moy + (int64_t)d0 * 64;
        // the group DG further, of this tile or the next, is copied into the slots these
        // chunks leave, while their steps wait for one another
        const int gi = d0 >> 2;
        if (gi + DG >= NG && !next_known) {
          unsigned w;
          if (peek(n + 1, w)) {
            next_known = true;
            Tile t1;
            if (w != kNoTile && tile_of(w, t1)) nc0 = ((int64_t)t1.id * kSweepWarps + cw) * NC;
          }
        }
        const SweepAhead go = sweep_ahead(gi, NC, DG, ahead, nc0 >= 0);
        if (go.next && go.chunks) ahead++;
        const int64_t cf = go.chunks ? chunk_at(go.next ? nc0 : c0, 4 * go.group) : c0;
        const int64_t fv = cf * 128 + lane * kLane, ff = cf * (Op::FS * 128) + lane * kLane;
        // What the next group's entries hold: asked for in the first chunk, looked at after the
        // last, since the answer comes from another block.  Their consumers took the last values
        // there two groups ago, unless they are late.
        RingWords look_nx, look_ny;
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int d = d0 + i;
          const bool live = kMain || d < NC;
          const int slot = (sbase + i) & (D - 1);
          const bool on = i < go.chunks;
          const int64_t av = fv + kDir * i * 128, af = ff + kDir * i * (Op::FS * 128);
          if (i == 0) {
            look_nx = ring_look<T>(look_x + nxt * kSlotX);
            look_ny = ring_look<T>(look_y + nxt * kSlotY);
          }
          if (live) {
            // the neighbours' boundary values, x entry d + 2 and y entry d + 1, and this
            // chunk's inputs.  (Fetching the next chunk's in the shadow of this one's
            // shuffles instead measured 5% slower: they share the shuffles' pipe.)
            Quad<T> xq, yq, v[NV];
            const bool take_x = has_x && (kMain || d < NC - 2), take_y = has_y && (kMain || d < NC - 1);
            take(take_x, i < 2 ? rxa + (i + 2) * kSlotX : rxb + (i - 2) * kSlotX, take_y,
                 i < 3 ? rya + (i + 1) * kSlotY : ryb, xq, yq, [&] {
                   cp_async_wait<D - 1>();  // one group of copies is committed per chunk
#pragma unroll
                   for (int k = 0; k < NV; k++) v[k] = chunk_load(stage + (slot * NV + k) * 128);
                 });

            if (!kMain && !take_x) xq = Quad<T>{};
            if (!kMain && !take_y) yq = Quad<T>{};
            const T xin[4] = {xc, xq.e[0], xq.e[1], xq.e[2]}, yin[4] = {yc, yq.e[0], yq.e[1], yq.e[2]};
            xc = xq.e[3];
            yc = yq.e[3];
            Quad<T> val;
            T o[NO][4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
              const int e = FWD ? j : 3 - j;
              T vv[NV], ov[NO];
#pragma unroll
              for (int k = 0; k < NV; k++) vv[k] = v[k].e[e];
              const T xs = FWD ? __shfl_up_sync(kFull, prev, 1) : __shfl_down_sync(kFull, prev, 1);
              const T ys = FWD ? __shfl_up_sync(kFull, prev, 8) : __shfl_down_sync(kFull, prev, 8);
              prev = op.step(vv, from_x ? xin[j] : xs, from_y ? yin[j] : ys, prev, ov, acc);
              val.e[j] = prev;
#pragma unroll
              for (int k = 0; k < NO; k++) o[k][e] = ov[k];
              // into the slot this chunk's inputs came from
              if (j == 0) copy(av, af, slot, on);
            }
            // until the words that this group's boundary values go to are empty
            if (i == 0 && held) {
              for (int spins = 0;;) {
                const uint32_t hx = ring_look<T>(look_x + cur * kSlotX).held(kEmpty),
                               hy = ring_look<T>(look_y + cur * kSlotY).held(kEmpty);
                if (!__any_sync(kFull, (feeds_x & (hx != 0)) | (feeds_y & (hy != 0)))) break;
                if (!__all_sync(kFull, W.more(spins, lim))) break;
              }
              __syncwarp();  // one lane looked, another one stores
            }
            // hand the boundary on (entry d; x entry 0 is not needed)
            const bool ox = xlast & ((i > 0) | (d0 > 0));
            ring_give(oxa + i * kSlotX, val, ox & feeds_x);
            ring_give(oya + i * kSlotY, val, ylast & feeds_y);
            mb_store(bx + i * 32, val, ox & out_x);
            mb_store(by + i * 64, val, ylast & out_y);
#pragma unroll
            for (int k = 0; k < NO; k++) chunk_store(op.out[k] + (ato + kDir * i * (Op::OS * 128)), o[k]);
          } else {
            copy(av, af, slot, on);
          }
          if (i == 3) held = __any_sync(kFull, (rings_x & (look_nx.held(kEmpty) != 0)) | (rings_y & (look_ny.held(kEmpty) != 0)));
          cp_async_commit();
        }
        group++;
        cur = nxt;
        __syncwarp();
      };
      for (int gi = 0; gi < NG; gi++) {
        if (4 * gi + 3 < NC - 2)
          four_chunks(std::true_type{}, 4 * gi);
        else
          four_chunks(std::false_type{}, 4 * gi);
        if (publisher && gi >= pub_at && pub < 3) advance_ticket(n);
      }
      if (publisher)
        while (pub < 3) advance_ticket(n);
      // This tile's share of the dot product, summed in a fixed order whichever block
      // swept which tile.  FP64: per 32 x 8 columns (two tiles) a tree over the 32
      // columns of each row, then the rows in order, done by the last warp to finish;
      // the last bits of z.r decide the rounding of every later iterate, so this tree
      // is part of the result (see k_spmv).  FP32: beta is rounded to FP32.
      if constexpr (sizeof(T) == 8) {
        if (a.col_sums) {
          a.col_sums[(tid * kSweepWarps + cw) * 32 + lane] = acc;
          __threadfence();
          __syncwarp();
          const int Y = tid / g.ntx, X = tid - Y * g.ntx, X2 = X >> 1, t32 = Y * ((g.ntx + 1) >> 1) + X2;
          const bool other = nb & (X & 1 ? 1 : 2);  // the other tile of the pair is swept
          int done = 0;
          if (lane == 0) done = atomicAdd(&a.t32_count[t32], 1) + 1;
          if (__shfl_sync(kFull, done, 0) == (other ? 2 : 1) * kSweepWarps) {
            __threadfence();
            double S = 0.0, c[8];
            const int Xl = X2 * 2 + (lane >> 4);
#pragma unroll
            for (int r = 0; r < 8; r++)
              c[r] = Xl < g.ntx ? __ldcg(&a.col_sums[((Y * g.ntx + Xl) * kSweepWarps + (r >> 2) * 2 + ((lane >> 3) & 1)) * 32 +
                                                     (r & 3) * 8 + (lane & 7)])
                                : 0.0;
#pragma unroll
            for (int r = 0; r < 8; r++) S += warp_sum(c[r]);
            if (lane == 0) {
              a.t32_sums[t32] = S;
              a.t32_count[t32] = 0;
            }
          }
        }
      } else {
        acc = warp_sum(acc);
        if (lane == 0) a.tile_partials[tid * kSweepWarps + cw] = acc;
      }
    }
    cp_async_wait<0>();
  }
  cluster_sync();  // nothing of this block's shared memory is accessed any more
  // exit accounting: the last block reduces the shares, runs the finalizer and
  // resets the counters
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_misc[1] = atomicAdd(a.exits, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (s_misc[1]) {
    double* sums = reinterpret_cast<double*>(dyn + SM::sums);
    __threadfence();
    double S = 0.0;
    if constexpr (sizeof(T) == 8) {
      // lane l sums the 32 x 8 tiles l, l + 32, ... in order, then a fixed tree
      if (a.fin_kind != 0 && a.col_sums && warp == 0) {
        const int n = ((g.ntx + 1) >> 1) * g.nty;
        for (int i = lane; i < n; i += 32) S += __ldcg(&a.t32_sums[i]);
        S = warp_sum(S);
      }
      if (lane == 0) sums[warp] = S;
    } else {
      if (a.fin_kind != 0)
        for (int i = threadIdx.x; i < g.ntiles() * kSweepWarps; i += kSweepThreads) S += __ldcg(&a.tile_partials[i]);
      S = warp_sum(S);
      if (lane == 0) sums[warp] = S;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      S = 0.0;
      for (int i = 0; i < kSweepThreads / 32; i++) S += sums[i];
      *a.ticket = 0;
      *a.exits = 0;
      if (a.fin_kind != 0) finalize(a.fin_kind, a.sc, S, 0.0);
      if (a.sc->err & DEV_ERR_TIMEOUT) a.sc->done = DONE_BREAKDOWN;
      __threadfence();
    }
  }
}

// One block per SM (more than half of its shared memory): two, with half the
// registers and stages each, measured 10-20% slower at 256^3 (FP64 forward sweep
// 284 us against 221) and no faster at 128^3.
template <class T, class Op>
constexpr int sweep_smem() {
  return SweepSmem<T, Op::NX + Op::NF>::bytes > 120 * 1024 ? SweepSmem<T, Op::NX + Op::NF>::bytes : 120 * 1024;
}
template <class T, bool FWD, class Op>
void sweep_set_attr() {
  cudaFuncSetAttribute(k_sweep<T, FWD, Op>, cudaFuncAttributeMaxDynamicSharedMemorySize, sweep_smem<T, Op>());
  cudaFuncSetAttribute(k_sweep<T, FWD, Op>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}
template <class T, bool FWD, class Op>
cudaLaunchConfig_t sweep_config(cudaLaunchAttribute* at, int clusters, int size, cudaStream_t st) {
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = size;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(clusters * size);
  cfg.blockDim = dim3(kSweepThreads);
  cfg.dynamicSmemBytes = sweep_smem<T, Op>();
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}
// Clusters of `size` blocks the GPU can hold at once (0: none).
template <class T, bool FWD, class Op>
int sweep_max_clusters(int size) {
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = sweep_config<T, FWD, Op>(&at, 1, size, nullptr);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k_sweep<T, FWD, Op>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}
template <class T, bool FWD, class Op>
void launch_sweep(const SweepArgs& a, const Op& op, cudaStream_t st, int clusters) {
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = sweep_config<T, FWD, Op>(&at, clusters, a.cx * a.cy, st);
  cudaLaunchKernelEx(&cfg, k_sweep<T, FWD, Op>, a, op);
}

// Fill the mailboxes with the sentinel (at allocation and after an error).
template <class T>
__global__ void k_mb_reset(int64_t quads, T* mb) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < quads; e += stride)
    mb_store(mb + 4 * e, sentinel_quad<T>());
}

}  // namespace
}  // namespace sc
