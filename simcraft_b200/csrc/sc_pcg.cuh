// sc_pcg.cuh -- MIC(0)-preconditioned CG pressure solver (FP64 and mixed FP32/FP64).
//
// Host-side interface of the solver behind CgSolver3D::solve
// (FluidSim/include/FluidSim/cpu/project-solver.h:100-131,
//  FluidSim/src/cpu/project-solver.cc:308-346) and
// ModifiedIncompleteCholesky3D::precond (project-solver.cc:230-306).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <string>
#include <vector>

#include "sc_common.cuh"

namespace sc {


struct Context {
  int device = 0;
  int sm_count = 148;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  // Bound of the device's spin-waits (wavefront mailboxes, grid barriers), in
  // polls; 0 selects each wait's default.  A wait that reaches it gives up and
  // the call returns SC_ERR_TIMEOUT.
  int wait_limit = 0;
  // Scratch of the stage functions, one block kept between calls (see ScratchLease).
  struct Arena {
    std::mutex m;
    void* base = nullptr;
    size_t cap = 0;
    cudaEvent_t done = nullptr;  // the last call's work on the block
  };
  mutable Arena arena;
  std::string last_error;
  int set_error(int code, const std::string& msg) {
    last_error = msg;
    return code;
  }
};

// One call's scratch on stream `st`.  A call takes the context's block, grown to what it
// needs, holds it while it enqueues its work and hands it on with an event that the next
// call waits for on its own stream, so calls from several threads and streams take turns.
// The block stays with the context: with an allocation per call the default pool, which
// keeps nothing across a wait for the GPU, mapped ~1 GB again each time (the transfers of
// 4.2M particles: 12 ms a call, 2 of them work).  It goes back when the context and its
// handles are destroyed.  kScratchKeep bounds what an idle context may hold, 1% of the
// GPU's memory: a P2G takes 60 bytes a particle and 202 a cell (16.8M particles on 128^3
// cells 1.4 GB), G2P and reconstruct 60 and 12.  Above it, and under stream capture, the
// call allocates and frees its own.
constexpr size_t kScratchKeep = (size_t)2 << 30;
class ScratchLease {
 public:
  ScratchLease(const Context& ctx, size_t bytes, cudaStream_t st) : st_(st), lock_(ctx.arena.m, std::defer_lock) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    const bool known = cudaStreamIsCapturing(st, &cap) == cudaSuccess;
    if (!known) cudaGetLastError();
    if (!known || cap != cudaStreamCaptureStatusNone || !ctx.arena.done || bytes > kScratchKeep) {
      if (cudaMallocAsync(&own_, bytes, st) == cudaSuccess) at_ = (char*)own_;
      return;
    }
    lock_.lock();
    Context::Arena& a = ctx.arena;
    if (cudaStreamWaitEvent(st, a.done, 0) != cudaSuccess) return;
    held_ = &a;
    if (a.cap < bytes) {
      if (a.base) cudaFreeAsync(a.base, st);
      a.base = nullptr;
      a.cap = 0;
      const size_t want = (bytes + ((size_t)1 << 20) - 1) >> 20 << 20;
      if (cudaMallocAsync(&a.base, want, st) != cudaSuccess) {
        a.base = nullptr;
        return;
      }
      a.cap = want;
    }
    at_ = (char*)a.base;
  }
  ~ScratchLease() {
    if (own_) cudaFreeAsync(own_, st_);
    if (held_) cudaEventRecord(held_->done, st_);
  }
  ScratchLease(const ScratchLease&) = delete;
  ScratchLease& operator=(const ScratchLease&) = delete;
  bool ok() const { return at_ != nullptr; }
  static size_t padded(size_t bytes) { return (bytes + 255) & ~(size_t)255; }
  // The next `bytes` of the block; the sum of padded(bytes) is what the lease was made for.
  template <class T>
  void take(T** p, size_t bytes) {
    *p = (T*)at_;
    at_ += padded(bytes);
  }

 private:
  cudaStream_t st_;
  std::unique_lock<std::mutex> lock_;
  Context::Arena* held_ = nullptr;
  void* own_ = nullptr;
  char* at_ = nullptr;
};

enum { CRIT_ABS_LINF = 0, CRIT_REL_L2 = 1 };
enum { PREC_FP64 = 0, PREC_MIXED = 1 };
enum { INNER_PCG = 0, INNER_EISENSTAT = 1 };
enum { DONE_RUNNING = 0, DONE_CONVERGED = 1, DONE_MAXITER = 2, DONE_BREAKDOWN = 3 };

struct PcgOptions {
  double tol = 1e-6;       // project-solver.h:129
  int max_iter = 300;      // project-solver.h:130
  int criterion = CRIT_ABS_LINF;
  int precision = PREC_FP64;
  double tau = 0.97, sigma = 0.25;  // project-solver.h:83-84
  double inner_rtol = 1e-4;  // mixed: relative reduction asked of each FP32 inner solve
  int max_outer = 50;        // mixed: defect corrections (FP64 residual replacements)
  int chunk = 8;             // PCG iterations per CUDA-graph launch
  int check_symmetry = 0;    // verify Right/Up/Front == shifted Left/Down/Back
  int true_residual = 1;     // recompute ||b - A p|| in FP64 at the end
  int inner_method = INNER_EISENSTAT;  // mixed: iteration of the FP32 inner solve
  double reliable_delta = 0.1;  // mixed, Eisenstat: split-residual reduction between FP64 replacements
};

struct PcgStats {
  int iterations = 0;        // the reference's `iter` (FP64); total inner iterations (mixed)
  int outer = 0;             // mixed: defect-correction passes
  int status = 0;            // DONE_* of the final (inner) solve
  double residual = 0;       // stopping measure at exit (recurrence residual)
  double true_rel_l2 = 0;    // ||b - A p||_2 / ||b||_2 in FP64
  double true_linf = 0;      // ||b - A p||_inf in FP64
  double ms = 0;             // device time of the solve (events)
  double sym_err = 0;        // max |A_R(p) - A_L(p+x)| etc. when checked
  unsigned device_flags = 0; // DEV_ERR_* bits raised on the device
  int64_t kernel_launches = 0;  // kernels launched by the solve (graph nodes counted)
};

// Device scalars shared by the kernels of one PCG run.
struct PcgScalars {
  double sigma, alpha, beta;
  double res, bnorm, tol, rscale;
  double rn2, rinf, sdotz;
  int iter, max_iter, done, criterion;
  unsigned err;
  unsigned count;  // last-block counter
  int first;       // 1 until the first preconditioner application has set sigma
  int spin_limit;  // polls before a sweep's wait gives up (0: the default bound)
};

template <class T>
struct SysArrays {  // one precision's copy of everything the PCG iterates on
  T *adiag = nullptr, *al = nullptr, *ad = nullptr, *ab = nullptr;  // the matrix (Tiled); the rest in the SweepLayout
  T *fwd = nullptr, *bwd = nullptr;  // the sweeps' factor streams (sc_sweep.cuh)
  T *r = nullptr, *p = nullptr, *z = nullptr, *s = nullptr, *q = nullptr, *Az = nullptr;
};

class PcgSolver {
 public:
  // PivotOp's inputs (SweepLayout): diagonal, lower couplings, neighbour products
  struct PivotIn {
    double* a[7];
  };
  PcgSolver(Context* ctx, int nx, int ny, int nz, const PcgOptions& opt);
  ~PcgSolver();
  int status() const { return init_status_; }
  // Load a system given in the reference layout (6 neighbour arrays, Left..Back
  // order of project-solver.cc:7-14).  `device` selects device or host pointers.
  int upload(const double* adiag, const double* const an[6], const double* rhs,
             const uint8_t* active, bool device);
  // Replace only the right-hand side (reference layout).
  int upload_rhs(const double* rhs, bool device);
  int solve(PcgStats* st);
  int download_pressure(double* pg, bool device);
  // ModifiedIncompleteCholesky3D::precond on the uploaded system: z = M^-1 r
  // (reference layout in and out, device pointers).
  int precond_only(const double* r, double* z);
  // applyCompressedMatrix on the uploaded system (device pointers, reference layout).
  int apply_only(const double* x, double* b);
  // Device time per launch of each kernel class (see sc_pcg_time_kernels).
  int time_kernels(int reps, double* ms);

  const Tiled& geom() const { return g_; }
  uint64_t launches() const { return launches_; }
  // Direct access for in-device producers (FLIP buildSystem writes these).
  double* adiag64() { return d64_.adiag; }
  double* al64() { return d64_.al; }
  double* ad64() { return d64_.ad; }
  double* ab64() { return d64_.ab; }
  double* rhs64() { return rhs_; }
  uint8_t* active() { return active_; }
  double* pressure64() { return press_; }
  // Called after a producer wrote adiag/al/ad/ab/active/rhs in tiled layout.
  void mark_system_changed() { pivots_valid_ = false; }
  void set_options(const PcgOptions& o) { opt_ = o; }
  const PcgOptions& options() const { return opt_; }

 private:
  int ensure_pivots();
  int ensure_matrix32();
  PivotIn pivot_in() const;
  // eis: Eisenstat iteration (FP32 inner solve of the mixed path only)
  template <class T>
  int run_pcg(SysArrays<T>& A, double tol, int criterion, int max_iter, bool scale_rhs,
              PcgStats* st, bool eis = false);
  int solve_fp64(PcgStats* st);
  int solve_mixed(PcgStats* st);
  int solve_mixed_reliable(PcgStats* st);
  template <class T>
  int ensure_graph(SysArrays<T>& A, bool eis);
  int true_residual(PcgStats* st);
  template <class T>
  void launch_iteration(SysArrays<T>& A, bool eis);
  template <class T>
  void launch_spmv(SysArrays<T>& A, cudaStream_t st, int use_skip);
  int check_dev_error(const char* where);
  // After a wavefront wait gave up: refill the mailboxes with the sentinel
  // (an aborted consumer leaves entries unconsumed), clear the status word and
  // drop the pivots, so the next solve starts from a clean state.
  int recover_after_timeout();
  int spin_limit() const;
  int pivot_limit_ = 0;  // host copy of the bound uploaded for the pivot sweep
  // Per tile: any active cell (set with the pivots); the sweeps of the
  // iterations visit only those tiles.
  uint8_t* tile_act_ = nullptr;
  void select_active_tiles();
  void choose_clusters();
  struct SweepPlan;  // what a sweep launch needs beside its operands
  SweepPlan sweep(bool f32, int use_skip, int fin, bool all_tiles = false) const;
  int ensure_host_stage();
  double* hstage_ = nullptr;     // staging of the host-array entry points (N doubles)
  uint8_t* hstage_act_ = nullptr;  // and of the active flags (N bytes)

  Context* ctx_;
  PcgOptions opt_;
  Tiled g_;
  SweepLayout sg_;
  int init_status_ = 0;
  bool pivots_valid_ = false;
  bool have_f32_ = false;
  bool matrix32_valid_ = false;  // the FP32 matrix is that of the pivots
  int nblocks_ = 0;     // elementwise grid
  SysArrays<double> d64_;
  SysArrays<float> d32_;
  // FP64, Tiled layout: the right-hand side, the solution, and the mixed solve's residual
  double *rhs_ = nullptr, *press_ = nullptr, *rres_ = nullptr;
  uint8_t* active_ = nullptr;
  double* partials_ = nullptr;  // 2 per block
  double* tile_partials_ = nullptr;
  PcgScalars* sc_ = nullptr;
  PcgScalars* sc_host_ = nullptr;  // pinned
  int* ticket_ = nullptr;  // sweep tickets and exit count (reset by each sweep's last block)
  // tiles in the sweeps' dependency order, after a header entry holding their
  // count: every tile (pivot sweep), and the tiles with an active cell
  int2 *order_all_ = nullptr, *order_act_ = nullptr;
  // the sweeps' cluster shape in tiles, clusters per launch, and the same lists of
  // cluster tiles
  int cl_x_ = 1, cl_y_ = 1, cl_grid_ = 1;
  int2 *order_cl_all_ = nullptr, *order_cl_act_ = nullptr;
  uint8_t *bits_all_ = nullptr, *bits_act_ = nullptr;  // SweepArgs::bits of these
  int2 *order_t32_all_ = nullptr, *order_t32_act_ = nullptr;  // of Tiled tiles
  // the FP64 sweep's dot product: per column, per Tiled tile, warps that are done
  double *col_sums_ = nullptr, *t32_sums_ = nullptr;
  int* t32_count_ = nullptr;
  // sweep mailboxes (per consumer tile), FP64 and FP32
  double *mbx64_ = nullptr, *mby64_ = nullptr;
  float *mbx32_ = nullptr, *mby32_ = nullptr;
  void reset_mailboxes(bool f32);
  std::vector<void*> allocs_;
  cudaEvent_t ev0_ = nullptr, ev1_ = nullptr;    // chunk polling
  cudaEvent_t evt0_ = nullptr, evt1_ = nullptr;  // solve timing
  double sym_err_ = 0.0;
  double inner_scale_ = 1.0;
  PcgScalars last_{};
  uint64_t launches_ = 0;  // kernels launched so far (graph nodes counted)
  // graphs: one chunk of iterations per precision
  cudaGraphExec_t graph64_ = nullptr, graph32_ = nullptr, graph32e_ = nullptr;
  template <class T>
  cudaGraphExec_t& graph_for(bool eis);
};

// Allocation-free ModifiedIncompleteCholesky3D::precond on device arrays in the
// reference layout, using a static device array as scratch (sc_pcg.cu).
int mic_precond_noalloc(cudaStream_t st, int device, int sm_count, int nx, int ny, int nz,
                        const double* adiag, const double* const* an, const double* r,
                        const uint8_t* active, double* z, double tau, double sigma,
                        std::string* msg);

}  // namespace sc
