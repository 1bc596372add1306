// xg_lu.h — the sparse LU of the Newton solve: host symbolic analysis
// (lu_symbolic.cpp) shared with the device refactor/solve (lu_kernels.cu).
//
// The reference factors the Jacobian with KLU through Amesos
// (N_LAS_AmesosSolver.C:231-492): one symbolic analysis per matrix pattern,
// a numeric factorisation with partial pivoting per Newton iteration, then
// the triangular solves.  Here the analysis runs once on the host: an
// approximate-minimum-degree column order, then a left-looking partial-pivot
// factorisation of the first matrix that fixes the row (pivot) order and the
// filled L\U pattern.  Every later factorisation reuses that pivot order and
// pattern and runs on the GPU.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "xg.h"

namespace xg {

struct LuSymbolic {
  int n = 0;
  int64_t nnz_a = 0;
  // B = A(P, Q): row k of B is row P[k] of A, column j of B is column Q[j].
  std::vector<int> P, Q;
  // Filled pattern of L\U of B, row-wise (CSR), columns ascending in each
  // row; L strictly left of the diagonal (unit diagonal implied), U from the
  // diagonal on.
  std::vector<int> rp, ci, diag;
  std::vector<int> lu2a;     // LU position -> CSR index of the A entry, or -1 (fill)
  double refactor_flops = 0;  // multiply-adds + divides of one refactorisation
  double solve_flops = 0;     // multiply-adds of one forward + backward solve
  int levels = 0;             // longest row dependency chain of the factorisation
  int max_width = 0;          // rows in the widest level of that chain
  int n_dense = 0;            // rows/columns ordered last as dense
  double min_pivot = 0, max_pivot = 0;  // |U(k,k)| range of the analysed matrix
  int ordering = 0;           // column order: 0 minimum degree, 1 nested dissection
  // Update schedule of the refactorisation (lu_build_updates): for row i, its
  // L entries p in ascending column k, and for each the entries q of U row k
  // right of the diagonal in ascending column, upos holds the position in
  // row i that U(k, ci[q]) updates.  urp[i] is where row i's updates start.
  std::vector<int64_t> urp;
  std::vector<int> upos;
};

// Ordering choice: nested dissection is tried when minimum degree leaves a
// dependency chain longer than kNdMinLevels rows with fewer than
// kNdMaxRowsPerLevel rows per level on average (a 60-stage chain: 61 levels in
// minimum-degree order, refactor and solve 85 us, 7 levels and 27 us in the
// other); parts of at most kNdLeaf vertices are ordered by minimum degree.  The refactorisation time model
// charges kLuLevelSeconds per dependent level and kLuFlopSeconds per
// multiply-add.
constexpr int kNdMinLevels = 16;
constexpr double kNdMaxRowsPerLevel = 8.0;  // and minimum degree averages fewer rows per level
constexpr int kNdLeaf = 4;  // 1,000-stage chain: 12 row levels against 22 with 16, the same fill
constexpr double kLuLevelSeconds = 2e-6;
constexpr double kLuFlopSeconds = 2e-10;
double lu_model_seconds(const LuSymbolic &S);

// Nested-dissection order of the graph of A + A^T (diagonal ignored).
std::vector<int> nd_order(int n, const int *rp, const int *ci, int leaf, int *n_dense);

// Approximate minimum degree order of the graph of A + A^T (diagonal
// ignored).  Returns the elimination order: order[k] = the k-th unknown.
std::vector<int> amd_order(int n, const int *rp, const int *ci, int *n_dense);

// Ordering + pivoting factorisation of A (CSR, n x n) with threshold partial
// pivoting (diagonal preferred when |a_diag| >= pivot_tol * max|column|).
// ordering: 0 minimum degree, 1 nested dissection, -1 chooses (see
// kNdMinLevels; XG_LU_ORDER=amd|nd in the environment overrides that choice).
// Returns 0, or -1 with *err set when A is structurally or numerically
// singular.
int lu_analyze(int n, const int *rp, const int *ci, const double *val, double pivot_tol,
               LuSymbolic *out, std::string *err, int ordering = -1);

// Fills the update schedule (urp, upos) from the L\U pattern; false if an
// update falls outside the pattern (cannot happen for a pattern lu_analyze
// made).
bool lu_build_updates(LuSymbolic &S);

// The elimination of a small factor entry by entry (lu_entries.cuh), as one
// image of 32-bit words.  Its head says where each part starts; a bound list
// holds, per level, where its short and its long members start.
constexpr unsigned kEntryU = 0, kEntryL = 1, kEntryPivot = 2, kEntryNone = 3;
constexpr int kEntryLong = 12;  // pairs or row entries a thread sums; longer ones take a warp
struct LuEntriesHead {
  int words = 0, solve0 = 0, both = 0;  // image; solve-only part [solve0, words); factor and solve [0, both)
  int factor = 0;                       // factor only [0, factor)
  int levels = 0, ulevels = 0, slevels = 0;
  int n_work = 0, n_pair = 0, max_width = 0;
  int ebound = 0, work = 0, pair = 0;   // entries: {position | row or column << 16 | kind << 30,
                                        // first pair | pairs << 16}; pairs {L position | U position << 16}
  int fbound = 0, frow = 0;             // forward rows by entry level
  int ci = 0, rp = 0, diag = 0;         // the pattern in 16 bits
  int ubound = 0, urow = 0;             // backward rows
  int sbound = 0, srow = 0;             // forward rows by row level (a solve on its own)
};
struct LuEntries {
  LuEntriesHead head;
  std::vector<uint32_t> image;
};
// Fills the image from the pattern and the update schedule (lu_build_updates);
// false when it needs more than 16-bit positions (65,535 entries or pairs,
// 16,383 rows).
bool lu_build_entries(const LuSymbolic &S, LuEntries *E);

// xg_lu_analyze for a transient, which does not read xg_lu_info: small
// factors with a solve chain may take the multifrontal path too.
int lu_analyze_transient(xg_ctx *ctx, int n, const int *host_rowptr, const int *host_colidx,
                         const double *host_values, int precision, xg_lu **out);

// Device address of an LU's status word (bits as xg_lu_status reports), for
// callers that read it back together with other results.
const unsigned *lu_status_device(const xg_lu *lu);

}  // namespace xg
