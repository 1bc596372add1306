// lu_front.h — multifrontal plan of a large Newton matrix (host).
//
// The row-wise grid path of lu_kernels.cu pays an L2 round trip per row of
// the longest dependency chain, thousands of them on a power grid or a block
// of logic.  The multifrontal method (Duff and Reid, "The multifrontal
// solution of indefinite sparse symmetric linear systems", ACM TOMS 9(3),
// 1983; on the pattern of B + B^T as in Amestoy, Duff and L'Excellent,
// "Multifrontal parallel distributed symmetric and unsymmetric solvers",
// CMAME 184, 2000) turns the same elimination into a tree of small dense
// matrices: a front holds the rows and columns of its pivots and of the
// border they touch, takes its children's Schur complements and its own
// entries of A, eliminates its pivots and leaves its own Schur complement to
// its parent.  Fronts of one tree level are independent, and nested
// dissection keeps the tree a dozen or two levels deep.
#pragma once

#include <cstdint>
#include <vector>

#include "xg_lu.h"

namespace xg {

constexpr int kFrontMax = 512;          // rows of the largest front the kernels take
constexpr int kFrontMiddle = 64, kFrontLow = 32;  // rows that part a level's fronts into size classes
constexpr int kFrontDouble = 48;         // rows up to which FP32 factors' fronts are eliminated in FP64
constexpr int kFrontMaxChildren = 512;  // children of a front (a CTA adds them in turn)

// Rows of B solved outside the tree.  A row with one entry left (a source's
// branch equation) gives its unknown before the tree, a column with one
// entry left (a source's current) after it; taking one out can leave others.
// Rows are listed round by round; a row of the list reads only unknowns of
// earlier rounds (before the tree) or of the tree and later-taken rounds
// (after it, where the rounds are in solving order).
struct FrontRows {
  std::vector<int> row;              // B row (= its unknown) per place
  std::vector<int> diag;             // its pivot's A entry
  std::vector<int64_t> ptr;          // its other entries: [ptr[i], ptr[i + 1])
  std::vector<int> col, a;           // unknown (B column), A entry
  std::vector<int> round;            // round r is [round[2r], round[2r + 2]); its rows longer than
                                     // kFrontLongRow end at round[2r + 1] and come first
};
constexpr int kFrontLongRow = 64;

struct Front {
  int p = 0, m = 0;                  // pivots; rows (pivots, then the border)
  int level = 0;                     // height in the tree, leaves 0
  int parent = -1;
  int64_t idx = 0;                   // its m unknowns in FrontPlan::idx
  int child0 = 0, child1 = 0;        // children in FrontPlan::child
  int64_t map = 0;                   // its border's places in its parent, FrontPlan::map
  int64_t acol = 0;                  // its na entries of A, FrontPlan::apos and aidx
  int na = 0;
  int64_t lo = 0, uo = 0, co = 0;    // factor (m x p), U right of it (p x b) and Schur complement
                                     // (b x b), all column by column
  int64_t pv = 0, bv = 0;            // its places in vectors of pivots / of border values
  int ctas = 1;                      // CTAs that factor it (set by front_create)
};

// Multiply-adds of eliminating p pivots of an m-row front.
inline double front_work(double p, double m) {
  const double b = m - p;
  return (m * m * m - b * b * b) / 3.0;
}

struct FrontPlan {
  int n = 0;
  std::vector<int> Q;                // B = A(P, Q): P as analysed, Q[k] the column paired with row P[k]
  std::vector<Front> front;          // by level, then size class, then work, most first
  std::vector<int> level;            // level l is front[level[l]] .. front[level[l + 1]]
  std::vector<int> idx, map;
  std::vector<int> child;            // child fronts
  std::vector<int64_t> inv;          // per child: where its inverse map starts in inv_map
  std::vector<int> inv_map;          // per child, per row of the parent: its border row or -1
  std::vector<int> apos, aidx;       // A entries by front and column: column * kFrontMax + row, A entry
  int64_t n_l = 0, n_u = 0, n_c = 0, n_pv = 0, n_bv = 0;
  FrontRows before, core, after;     // core: the tree's rows and their entries in `before` unknowns
  double flops = 0;                  // multiply-adds of the tree's eliminations
  double seconds = 0;                // modelled refactor and solve
};

// Plans the multifrontal elimination of A (rows in S's pivot order): its
// pivots (singletons first, then the diagonal, a transversal where that has
// gaps) and a nested-dissection order.  False when a row's columns do not
// ascend, A is structurally singular, or a front would exceed kFrontMax rows
// or kFrontMaxChildren children.
bool build_front_plan(const LuSymbolic &S, const int *rp, const int *ci, FrontPlan *plan);

// Device side (lu_front.cu).
struct FrontLu;
// Uploads the plan; nullptr when device memory runs out, a front is too large
// for shared memory or the device does not grant a launch its clusters.
FrontLu *front_create(const FrontPlan &plan, const LuSymbolic &S, int device, int precision);
void front_destroy(FrontLu *f);
// Refactors from dev_values (an FP64 copy goes to a_copy); status[0] collects
// status bits (1: zero or non-finite pivot, 2: a wait gave up after *limit
// polls), status[1] the first row with such a pivot.
int front_refactor(FrontLu *f, const double *dev_values, double *a_copy, int64_t nnz_a, unsigned *status,
                   const unsigned *limit, void *stream);
int front_solve(FrontLu *f, const double *a_copy, const double *b, double *x, unsigned *status, const unsigned *limit,
                void *stream);
// The largest |multiplier| of the last refactor (synchronises the stream).
int front_max_multiplier(FrontLu *f, double *out, void *stream);

}  // namespace xg
