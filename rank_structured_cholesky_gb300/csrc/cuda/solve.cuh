// Preconditioner apply x = (L L^T)^{-1} b with the GPU factor, in the
// permuted ordering (the caller keeps its vectors permuted).
//
// Same operator as FactorPreconditioner::solve -> FactorManager::solveSystem
// (src/rschol/solver/FactorPreconditioner.cpp:135-162,
// FactorManager.cpp:6245-6581, Supernode.cpp:4571-5250): interior nodes use
// their full factor panels (the rows the reference re-derives through
// A_{rest,I} L_I^{-T} L_I^{-1} are stored explicitly), compressed nodes use
// the (HODLR-expanded) dense L11 and the V U^T off-diagonal.
//
// Every supernode is applied through products formed once per factorisation,
// so that no triangular chain lies between the levels of the tree:
//   interior    X = L11^{-1}, G = L21 X:
//               up u = (children's rows) - G f, y = X f; down x = X^T y - G^T x_R
//   compressed  X = L11^{-1}, W = X^T U (L21 = V U^T):
//               up z = W^T f, u = -V z; across t = X^T (X f);
//               down s = V^T x_R, x = t - W s
// (the same operator up to rounding: L11^{-T} (L11^{-1} f - L21^T x_R)).  The inverse
// of the triangle, used from both sides, leaves residuals of the rounding level as
// substitutions do; S = (L11 L11^T)^{-1}, one product instead of two, leaves the
// block's condition number in them (dense block of 100, condition 1e10, b = A x of a
// random x, FP64: |b - A x| / |A| |x| 6.9e-9 with S, 3.2e-16 with X, 1.7e-16 by
// substitution), and is some 8 % quicker where an application is all latency (2D
// 40 x 37 FP64 91 against 100 us, 193 x 187 171 against 189, in groups of eight).
// X by inverted 64 x 64 diagonal blocks and recursive doubling X_BA = -X_BB
// L_BA X_AA with batched GEMMs; W, and G above 64 columns, by batched GEMMs; G of
// the small supernodes by one kernel.
// One persistent launch works the whole application off as a list of items in
// topological order (solve.cu).  Every sum has a fixed order and no atomics
// touch the numbers: results are bitwise reproducible.
#pragma once
#include <cuda_runtime.h>

#include <stdexcept>
#include <array>
#include <map>
#include <vector>

#include "factor.cuh"

namespace rschol {

constexpr int SOLVE_RB = 64;   // rows per compressed row block

template <class T>
struct SNode {
  const T* L;       // interior: [L11; L21] panel; compressed: L11 (HODLR expanded)
  const T* V;       // compressed: m x r
  const T* U;       // compressed: n x r
  T* X;             // L11^{-1} (n x ldx, row-major, upper triangle zero)
  T* G;             // interior: L21 L11^{-1} (m x ldk)
  const T* W;       // compressed: X^T U (n x r)
  int ld, n, m, r, c0;
  int ldk, ldx;               // row strides of G, and of X (interior: the same)
  int uOff, tOff;             // update vector (interior: children's rows - G f, compressed: -V z), and
                              // y = X f of an interior supernode
  long long relOff;           // interior: target index in the parent front of each row
  long long cOff;             // compressed: first of its n+1 contribution-list offsets
};

struct SPull {       // contribution source of a compressed supernode (plan time)
  int src;           // source node
  int a0, a1;        // source rows mapping into this node's columns
  int kind;          // 0: interior root update vector, 1: compressed V z
};

struct RowBlock {    // one thread block's work: (supernode, row block)
  int node, b;
};

struct PackTile {    // a tile of X packed for the apply: rows from i0, columns from j0
  int node, i0, j0, cols, rows;
};

struct alignas(16) ApplyItem {   // one work item of an application
  const void* g0;   // its pieces of the factor ...
  const void* g1;
  int kind;
  int bytes0, bytes1;          // ... and their bytes to stage (0: read in place, or none)
  int desc, descBytes;         // descriptor: offset in the blob (ints), bytes to stage (0: read in place)
  int waits;                   // (counter, target) pairs at the descriptor's start
  int sig;                     // counter released when the item is done
  int count;                   // members of a group
  int shallow;                 // an item of a phase of few items (ticket draw)
  int desc2, desc2Bytes;       // a part of the descriptor that several items share
  int early;                   // waits that come first; the batched kernel has work between them and the others
};

template <class T>
struct DinvTask {    // invert one lower-triangular diagonal block (h x h, h <= 64)
  const T* L;
  int ld, h;
  int pad;           // D is pad x pad, zero outside the h x h lower triangle
  int ldD;           // row stride of D
  T* D;
};

enum { XS_SIMT = 0, XS_ROWS128, XS_TC };   // SIMT in square tiles or in tiles of 128 x 64, tensor cores
struct XStep {       // one batched GEMM launch (X = L11^{-1} doubling, W and G)
  long long off;
  int count, tiles;
  int kind;
  int bn = 64;       // tensor-core tile width of the launch
};

template <class T>
class SolveEngine {
 public:
  explicit SolveEngine(FactorEngine<T>& F);
  void plan();                           // after the factor plan
  // Queue the solve-side preprocessing of a fresh factor (inverted diagonal
  // blocks); returns its launches.
  int prepare(cudaStream_t s);
  // w (permuted, length n, device) := M^{-1} w, in place.
  void apply_inplace(double* d_w, cudaStream_t s);
  // Reads (synchronously) and clears the error word of the row-block waits:
  // 0, or 1 if a wait gave up (the result of that apply is undefined).
  int take_error(cudaStream_t s);
  // Batched apply: W (n x k, row-major: the k right-hand sides of a row are
  // contiguous) := M^{-1} W with one pass over the factor; k <=
  // batch_capacity().  take_error_batch: as take_error, for the batched path.
  void apply_batch(double* d_W, int k, cudaStream_t s);
  // Time the candidate launch shapes of every width class up to kmax on this
  // stream (run it while the GPU is otherwise quiet) and keep the fastest.
  void autotune_batch(int kmax, cudaStream_t s);
  // the shapes chosen for each width class so far: (class, blocks per SM, columns per pass, 0, 0, ms) rows
  std::vector<std::array<double, 6>> batch_tuning() const;
  int batch_capacity() const;
  int batch_slices(int kp) const;   // slices of columns of a batched application
  // bumped whenever the batched apply's buffers are reallocated or its
  // shapes retuned (a graph that captured an apply must then be captured again)
  long long batch_generation() const { return batchGen_; }
  int take_error_batch(cudaStream_t s);
  long long launches_per_apply() const { return launchesPerApply_; }
  double bytes_per_apply() const { return bytesPerApply_; }

 private:
  FactorEngine<T>& F_;
  std::vector<SNode<T>> nodes_;
  DevBuf dNodes_, dWu_, dW_;
  DevBuf dDinvTasks_, dZp_, dSp_, dIp_, dT_, dYp_, dXp_, dSync_;
  // the work items and their descriptors, the counters ([0] error word,
  // [1] ticket), the single-vector launch's shape
  DevBuf dItems_, dBlob_, dPackTiles_, dPacked_;
  int nPacks_ = 0;
  int nItems_ = 0, nSync_ = 0, sms_ = 1, grid_ = 1, fLen_ = 4, work_ = 0;
  size_t smem_ = 0;
  bool group_member(int s) const;
  void plan_items(const std::vector<int>& rel, const std::vector<long long>& cstart, const std::vector<int>& ents);
  DevBuf dG_, dXi_, dWc_, dOpsWork_;                // G and X of the interior, W of the compressed supernodes
  std::pair<long long, int> opsClass_[3];           // work of interior_ops_kernel per column class
  DevBuf dX_, dT1_, dXGemm_;          // X of the compressed supernodes, the doubling's temporaries and GEMM tasks
  std::vector<XStep> xSteps_;
  int nDinv_ = 0;
  void plan_inverse();                // GEMM schedule of X = L11^{-1}
  long long launchesPerApply_ = 0;
  double bytesPerApply_ = 0;
  // batched apply: work buffers sized for the widest block seen, and per width
  // class (columns rounded up to a power of two) the persistent blocks per SM
  // (fixed unless tuned by autotune_batch or, with RSCHOL_AUTOTUNE=1, on first
  // use); no choice changes any column's arithmetic
  struct BatchCfg {
    int blocks = 2;
    double ms = 0;   // the winning candidate's time (0: not timed)
  };
  const BatchCfg& config_for(int k, cudaStream_t s, bool tune);
  int width_class(int k) const;
  void apply_batch_cfg(double* W64, int k, cudaStream_t s, const BatchCfg& c);
  std::map<int, BatchCfg> tuned_;
  bool autotune_ = true;
  void plan_batch(int kp);
  int kAllocB_ = 0;
  long long batchGen_ = 0;
  DevBuf dWuB_, dTB_, dZpB_, dSpB_, dYpB_, dXpB_, dIpB_, dSyncB_, dWB_;
};

}  // namespace rschol
