// Whole PCG solves in one cooperative launch (persist.cu): every lane (one
// system with one right-hand side) is solved from b to x by a group of CTAs
// that synchronise among themselves.
#ifndef ISPM_PERSIST_H
#define ISPM_PERSIST_H

#include <cuda_runtime.h>

#include <vector>

#include "operator.h"

namespace ispm {

// A sliced-ELL operator as the persistent kernel walks it: fixed slice
// height, one column per stored index.  The lane's rows start at slice
// slice0; columns [col0, col0 + rows) are its own (others read as 0).
struct PersistOp {
  const unsigned *sp = nullptr;  // slice_ptr (diagonal positions are indexes into it)
  unsigned slice0 = 0;
  const unsigned *cols = nullptr;
  const void *elms = nullptr;
  unsigned log2h = 0;   // slice height
  unsigned col0 = 0;
  int diag = 0;         // diagonal blocks after the explicit columns
  float inv_scale = 1.f;
};

struct PersistLane {
  PersistOp A, A64, G, Ht;  // inner matrix, FP64 matrix, factor pair
  long long row0 = 0;       // the lane's first row in the vectors
  int rows = 0;             // padded rows (a multiple of 32)
  int n = 0;                // rows of b that are read (the others count as 0)
  int cta0 = 0, ncta = 1;   // its CTAs
};

// Rows a thread of the walk (4, 2, 1), or four threads a row.
enum PersistShape { kRow4, kRow2, kRow1, kQuarter };
// The shape for `rows` rows of about `width` entries on `threads` threads, the
// fewest rows a thread that leave each thread one turn; min_height: the
// shortest slice height of the operators.
PersistShape persist_shape(double rows, double threads, double width, unsigned min_height);

struct PersistKind {
  int inner = ISPM_F32;    // vectors and A
  bool pipelined = false;  // (FP64 only)
  bool factor_f16 = false; // FP16 factor values (FP32 vectors)
  PersistShape shape = kRow1;
  // sixteen entries' loads of a thread in flight, at most kPersistWideThreads
  // threads a CTA (against eight and 1024: 27-point mixed solves 0.98 / 1.11 ms
  // at 56^3, 1.50 / 1.64 ms at 72^3)
  bool wide = true;
};
constexpr int kPersistWideThreads = 640;

// What a lane's solve reports.
struct PersistOut {
  double bnorm, rel;
  int iterations, replacements, restarts, status;
  int n_history, pad;
};

constexpr long long kPersistWaitCycles = 2000000000LL;  // about a second

struct PersistParams {
  const PersistLane *lanes = nullptr;  // device; lanes of one group in a row
  const int *cta_lane = nullptr;       // CTA -> first lane of its group
  const int *lane_count = nullptr;     // lanes of that group, by first lane
  // inner vectors.  Classic: R, P, Q, D, Z, T and second ones of R and P;
  // pipelined: R, U, W, M, P, S, Q, Z, D, T
  void *vec[10] = {};
  double *r64 = nullptr;
  const double *b = nullptr;
  double *x = nullptr;
  double *part = nullptr;     // partial sums, kPersistParts per CTA
  unsigned *bar = nullptr;    // a count per lane (zeroed before a launch)
  int n_ctas = 0;
  int max_tiles = 0;          // tiles of the largest CTA share
  unsigned *abort = nullptr;  // set when a wait ran out (zeroed before a launch)
  PersistOut *out = nullptr;  // per lane
  double *history = nullptr;  // true relative residual of each phase (one lane only)
  int history_cap = 0;
  int have_prec = 1;
  int batch = 0;              // the batched solver's accounting of phases
  double tol = 0, ru2 = 0;
  int max_iters = 0, max_refinements = 0;
  long long wait_cycles = kPersistWaitCycles;  // longest wait of a CTA
};

// The operator as PersistOp, or false when its shape is not one the kernel
// walks.  row0: the first row (and column) of a system inside a stack.
bool persist_op(const Operator &op, long long row0, PersistOp &out);

// Tiles of a CTA's share of `rows` rows split over ncta CTAs.
int persist_tiles(const PersistKind &k, int rows, int ncta);
// The most CTAs of `threads` threads one launch may have (all resident at
// once) with room for max_tiles tile headers of each operator; 0 for a kind
// without a kernel or headers that do not fit.
int persist_capacity(const PersistKind &k, int threads, int max_tiles, int &ctas);
constexpr size_t kPersistMaxSmem = 96 * 1024;  // (the rest of an SM's 228 KB is L1 for x)
constexpr int kPersistParts = 6;
constexpr int kPersistMaxDiag = 32;            // diagonals of a slice

// One launch: cooperative, `ctas` CTAs of `threads` threads.  refused (and
// ISPM_OK, no launch and no error left): the CTAs cannot all be resident, where
// the process has a part of the SMs.  fault: what a test has the launch return.
int persist_launch(const PersistParams &p, const PersistKind &k, int ctas, int threads,
                   cudaStream_t s, cudaError_t fault, bool &refused);

// CTAs for lanes of the given work: shares proportional to it, at least one
// each, at most ctas in all and at most one per 32 rows; lanes beyond the
// CTAs queue in groups of one CTA.  Fills cta0 / ncta and returns the lane
// order (groups in a row), the CTA -> first lane table and the group sizes.
// Returns the CTAs used.
int persist_assign(std::vector<PersistLane> &lanes, const std::vector<double> &work, int ctas,
                   std::vector<int> &order, std::vector<int> &cta_lane,
                   std::vector<int> &lane_count);

// Largest per-iteration working set (matrices and vectors, bytes) a solve
// takes this way.  Per iteration, this way against the step kernels, us: 55 MB
// 30.9 / 47.0, 107 MB 43.3 / 52.7, 162 MB 67.1 / 66.3 (27-point FP32, 64^3 to
// 92^3), 138 MB 36.8 / 47.8 (27-point FP64, 64^3); beyond, the step kernels'
// four rows a thread and higher occupancy stream HBM better.  A batch's lanes read
// a system's matrix at their own pace, which the shared launches do tile by
// tile, so its line is lower.
constexpr double kPersistMaxBytes = 150e6;
constexpr double kPersistMaxBatchBytes = 100e6;

}  // namespace ispm

#endif
