// lu_front.cu — multifrontal refactorisation and solves of large Newton
// matrices on the GPU (plan: lu_front.h).
//
// A tree level is one launch.  front_factor keeps a whole front in shared
// memory, its columns dealt in blocks of 4 to the CTAs it takes: 1 to 16 of a
// cluster, which several fronts share when they are small.  The owner of the
// next pivot columns updates and eliminates them first, one warp taking the
// pivot rows lane to lane while the others bring the lower rows up to date,
// and signals the front's other CTAs through mbarriers in their shared
// memory; those fetch the columns while it goes on with its other columns.
// An FP64 instruction takes a sub-partition 66 cycles, dependent or not and
// however few lanes it has (77 with all four busy), so what counts is the
// number of warp instructions: the updates are dealt entry by entry over all
// lanes, and the pivots' serial chain (reciprocal, multiplier, update) is
// kept to the fewest.  The forward and backward solves are one launch that
// walks the tree by flags.
//
// Measured: the 253-row root of a 200x200 power grid in 259 us (429 with a
// barrier per pivot and every CTA of the front reading the owner's shared
// memory), a whole refactor and solve of that grid 1.84 ms, of 200,000 devices
// of logic 2.30 ms.
//
// Every sum has a fixed order: results repeat bit for bit.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

#include "lu_entries.cuh"
#include "lu_front.h"
#include "xg_internal.h"
#include "xg_launch.cuh"
#include "xg_smem.cuh"

namespace xg {
namespace {

// Pivot columns eliminated at a time, and the unit of dealing columns: an
// elimination costs a warp kNb (kNb + 1) / 2 FP64 instructions however many
// of its lanes have rows, and bringing a row up to date kNb^2, much of it on
// the pivots' serial chain; the hand-over between CTAs costs about 1,300
// cycles.
constexpr int kNb = 4;
constexpr int kMaxCtas = 16;       // of one front
constexpr size_t kSmemLimit = 225 * 1024, kSmemTarget = 56 * 1024;
constexpr int kFlowThreads = 128;

struct ChildDev {
  int64_t inv, co, bv, map;
  int b, front, own;
};

struct FrontDev {
  const Front *front;
  const ChildDev *child;
  const int *idx, *map, *inv_map, *apos, *aidx;
  const int *own, *own_at;        // a child's border columns by the CTA of its parent that holds them (border
                                  // column | local column << 16, beside map), and where each CTA's start
  const int *P, *Q;
  void *l, *u, *c;                // factors and Schur complements (T)
  void *rd, *y, *bv;              // reciprocal pivots, forward values, border sums (T)
  double *xk;                     // unknowns by B column
  unsigned *status;
};

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// The two halves of a barrier over the cluster; a block's shared memory may be
// touched by others only once it is known to have started, so a kernel that
// does passes one before.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
  cluster_arrive();
  cluster_wait();
}
// The kernels here follow one another closely (xg_launch.cuh), 15 to 30 a
// step.  Measured: 20x20 power grid 211 to 178 us, 60x60 577 to 537, 200x200
// 1,910 to 1,843, 200,000 devices of logic 2,375 to 2,296.  (Letting them start
// as soon as the blocks ahead have started fills SMs unevenly: the last two
// took 1,940 and 2,564 us.)
__device__ __forceinline__ unsigned smem_u32(const void *p) { return unsigned(__cvta_generic_to_shared(p)); }
// One arrival at an mbarrier of another CTA of the cluster (its address from
// remote()); what the caller saw or wrote before is visible to whoever sees it.
__device__ __forceinline__ void signal(unsigned remote_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
}
// Waits for the barrier's phase of this parity, at most `limit` polls.
__device__ __forceinline__ bool await(unsigned bar, unsigned parity, int limit) {
  for (int it = 0; it < limit; ++it) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// This CTA's shared address p, in CTA `rank` of the cluster.
__device__ __forceinline__ unsigned remote(const void *p, unsigned rank) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(unsigned(__cvta_generic_to_shared(p))), "r"(rank));
  return a;
}
// Four loads in flight at once from other CTAs' shared memory.
__device__ __forceinline__ void remote_load4(const unsigned (&a)[4], double (&v)[4]) {
  asm volatile(
      "ld.shared::cluster.f64 %0, [%4];\n ld.shared::cluster.f64 %1, [%5];\n"
      "ld.shared::cluster.f64 %2, [%6];\n ld.shared::cluster.f64 %3, [%7];"
      : "=&d"(v[0]), "=&d"(v[1]), "=&d"(v[2]), "=&d"(v[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3])
      : "memory");
}
__device__ __forceinline__ void remote_load4(const unsigned (&a)[4], float (&v)[4]) {
  asm volatile(
      "ld.shared::cluster.f32 %0, [%4];\n ld.shared::cluster.f32 %1, [%5];\n"
      "ld.shared::cluster.f32 %2, [%6];\n ld.shared::cluster.f32 %3, [%7];"
      : "=&f"(v[0]), "=&f"(v[1]), "=&f"(v[2]), "=&f"(v[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3])
      : "memory");
}

// Columns of an m-column front that CTA r of C holds.
__host__ __device__ inline int local_columns(int m, int r, int C) {
  const int blocks = (m + kNb - 1) / kNb, mine = blocks > r ? (blocks - r + C - 1) / C : 0;
  const bool last = mine > 0 && (blocks - 1) % C == r;
  return mine * kNb - (last ? blocks * kNb - m : 0);
}
// An odd column stride: lanes on consecutive columns touch different banks.
__host__ __device__ inline int column_stride(int m) { return m | 1; }

// Fronts of at most kFrontDouble rows are eliminated in FP64 whatever the
// factors are kept in: that is where FP32 arithmetic loses most, and the tree
// would be less accurate than the minimum-degree order.  Forward error after
// two refinements of FP32 factors, row by row / tree in FP32 / tree so: 50x30
// power grid 3.8e-14 / 6.0e-13 / 2.6e-15, 72x72 1.2e-14 / 2.4e-12 / 5.5e-15,
// 150x150 9.8e-13 / 1.0e-12 / 4.2e-14.  (At 32 rows it would still be five
// times the row-wise one, at 40 three times after one refinement.)  The
// refactors take 240 -> 288 us (72x72), 510 -> 567 us (20,000 devices of logic)
// and 915 -> 1,016 us (150,000); another refinement step would cost 105, 177
// and 308 us.
size_t factor_smem(int m, int C, size_t tsz) {
  if (m <= kFrontDouble) tsz = sizeof(double);
  const size_t ld = size_t(column_stride(m));
  return ((C > 1 ? kNb : 0) + size_t(local_columns(m, 0, C))) * ld * tsz + (kNb * kNb + kNb) * tsz;
}

__device__ __forceinline__ void report_pivot(unsigned *status, int row) {
  atomicOr(status, 1u);
  atomicMin(status + 1, unsigned(row));
}

// This CTA's place of column j, -1 if another CTA holds it.
__device__ __forceinline__ int local_column(int j, int r, int C) {
  const int b = j / kNb;
  if (C == 1) return j;
  return b % C == r ? (b / C) * kNb + j % kNb : -1;
}

// The columns this CTA holds, summed from A and the children's Schur
// complements.  All threads take a child at a time: of its columns those this
// CTA holds (FrontDev::own lists them), their entries in the order they lie
// in memory, kE loads of a thread in flight; a child's loads are issued
// before the one before it is added and a barrier passed.  What bounds it is
// a child's L2 round trip.  (Looking at every entry of a child for the few of
// 16 CTAs' columns took 104 us of the 410 us of a 253-row root; a warp per
// column, children in turn, 50 us for a single front of 32 rows.)
template <class W, class T>
__device__ void assemble(const FrontDev &d, const Front &f, const double *a, W *F, int ld, int ncl,
                         int r, int C) {
  const int tid = threadIdx.x, bd = blockDim.x;
  constexpr int kE = 8;
  int at[kE], at_next[kE];
  T v[kE], v_next[kE];
  int c = f.child0, from = 0;  // the next entries to load: `from` on of child c
  auto load = [&](int (&to)[kE], T (&val)[kE]) {
#pragma unroll
    for (int q = 0; q < kE; ++q) to[q] = -1;
    if (c >= f.child1) return;
    const ChildDev g = d.child[c];
    const int o0 = __ldg(d.own_at + g.own + r), o1 = __ldg(d.own_at + g.own + r + 1), b = g.b, n = (o1 - o0) * b;
    const T *s = (const T *)d.c + g.co;
    const int *map = d.map + g.map, *own = d.own + g.map + o0;
    const float inv = 1.0f / float(b);  // (entry + 1/2) / b: exact, as in update_rest
#pragma unroll
    for (int q = 0; q < kE; ++q) {
      const int k = from + q * bd + tid;
      if (k < n) {
        const int jj = int((float(k) + 0.5f) * inv), i = k - jj * b, o = __ldg(own + jj);
        to[q] = (o >> 16) * ld + __ldg(map + i);
        val[q] = __ldcg(s + (o & 0xffff) * b + i);
      }
    }
    from += kE * bd;
    if (from >= n) {
      from = 0;
      ++c;
    }
  };
  load(at, v);
  for (int e = tid; e < ncl * ld; e += bd) F[e] = W(0);
  __syncthreads();
  const int64_t e0 = f.acol, e1 = f.acol + f.na;
  for (int64_t e = e0 + tid; e < e1; e += bd) {
    const int to = __ldg(d.apos + e), lc = local_column(to / kFrontMax, r, C);
    if (lc >= 0) F[size_t(lc) * ld + to % kFrontMax] = W(a[__ldg(d.aidx + e)]);
  }
  __syncthreads();
  if (f.child0 == f.child1) return;
  for (;;) {
    const bool last = c >= f.child1, new_child = from == 0;
    load(at_next, v_next);
#pragma unroll
    for (int q = 0; q < kE; ++q) {
      if (at[q] >= 0) F[at[q]] += W(v[q]);
      at[q] = at_next[q];
      v[q] = v_next[q];
    }
    if (new_child) __syncthreads();
    if (last) break;
  }
}

// The pivot columns [k0, k0 + nb) that start at base are eliminated in two
// parts.  pivot_rows: one warp takes the rows [k0, k0 + 32) in registers, a
// row per lane, and passes pivot rows and reciprocals lane to lane (no
// barrier; a pivot costs its reciprocal's and two more FP64 latencies).  It
// leaves pivot rows (su) and reciprocals (sr) for ...
template <class T>
__device__ __forceinline__ void pivot_rows(T *base, int ld, int k0, int nb, int m, T *su, T *sr) {
  const int lane = threadIdx.x & 31, i = k0 + lane;
  const bool mine = i < m;
  T v[kNb], own = T(0);
#pragma unroll
  for (int q = 0; q < kNb; ++q) v[q] = q < nb && mine ? base[size_t(q) * ld + i] : T(0);
#pragma unroll
  for (int q = 0; q < kNb; ++q) {
    if (q < nb) {
      // no branches: a divergent one costs as much as an FP64 instruction,
      // and each is on the pivots' chain (rows above take a multiplier of 0)
      const T pivot = __shfl_sync(0xffffffffu, v[q], q);
      T u[kNb];
#pragma unroll
      for (int s = q + 1; s < kNb; ++s) u[s] = __shfl_sync(0xffffffffu, v[s], q);
      const T rc = pivot_reciprocal(pivot), t = v[q] * rc, l = lane > q ? t : T(0);
#pragma unroll
      for (int s = q + 1; s < kNb; ++s) v[s] -= l * u[s];
      v[q] = lane > q ? t : v[q];
      own = lane == q ? rc : own;
    }
  }
#pragma unroll
  for (int q = 0; q < kNb; ++q)
    if (q < nb && mine) base[size_t(q) * ld + i] = v[q];
  if (lane < nb) {
    sr[lane] = own;
#pragma unroll
    for (int q = 1; q < kNb; ++q)
      if (q > lane) su[lane * kNb + q] = v[q];
  }
}
// ... lower_rows: all warps take the rows from k0 + 32 on.
template <class T>
__device__ __forceinline__ void lower_rows(T *base, int ld, int k0, int nb, int m, const T *su, const T *sr) {
  for (int i = k0 + 32 + int(threadIdx.x); i < m; i += blockDim.x) {
    T v[kNb];
#pragma unroll
    for (int q = 0; q < kNb; ++q) v[q] = q < nb ? base[size_t(q) * ld + i] : T(0);
#pragma unroll
    for (int q = 0; q < kNb; ++q) {
      if (q < nb) {
        v[q] *= sr[q];
#pragma unroll
        for (int s = q + 1; s < kNb; ++s)
          if (s < nb) v[s] -= v[q] * su[q * kNb + s];
        base[size_t(q) * ld + i] = v[q];
      }
    }
  }
}

// Columns [l0, l1) of this CTA after the pivots [k0, k0 + nb), whose
// eliminated columns are pan: their U rows, a column per thread (t of n), ...
template <class T>
__device__ __forceinline__ void update_u(T *F, int ld, int l0, int l1, const T *pan, int k0, int nb, int t, int n) {
  for (int c = l0 + t; c < l1; c += n) {
    T *col = F + size_t(c) * ld + k0;
    T u[kNb];
#pragma unroll
    for (int q = 0; q < kNb; ++q) u[q] = q < nb ? col[q] : T(0);
#pragma unroll
    for (int q = 1; q < kNb; ++q) {
      if (q < nb) {
#pragma unroll
        for (int s = 0; s < q; ++s) u[q] -= pan[s * ld + k0 + q] * u[s];
        col[q] = u[q];
      }
    }
  }
}
// ... and the entries [e0, e1) of the rows below (column by column), two per
// thread at a time (their chains of kNb multiply-adds are independent).
template <class T>
__device__ __forceinline__ void update_rest(T *F, int ld, int l0, const T *pan, int k0, int nb, int m, int e0, int e1,
                                            int t, int n) {
  const int i0 = k0 + nb, rem = m - i0;
  const float inv = 1.0f / float(rem);  // (entry + 1/2) / rem: exact below 2^18 entries of 512 rows
  for (int e = e0 + t; e < e1; e += 2 * n) {
    const int e2 = e + n < e1 ? e + n : e;
    const int c = int((float(e) + 0.5f) * inv), i = i0 + (e - c * rem);
    const int c2 = int((float(e2) + 0.5f) * inv), i2 = i0 + (e2 - c2 * rem);
    T *col = F + size_t(l0 + c) * ld, *col2 = F + size_t(l0 + c2) * ld;
    T acc = col[i], acc2 = col2[i2];
    if (nb == kNb) {
#pragma unroll
      for (int q = 0; q < kNb; ++q) {
        acc -= pan[q * ld + i] * col[k0 + q];
        acc2 -= pan[q * ld + i2] * col2[k0 + q];
      }
    } else {
      for (int q = 0; q < nb; ++q) {
        acc -= pan[q * ld + i] * col[k0 + q];
        acc2 -= pan[q * ld + i2] * col2[k0 + q];
      }
    }
    col[i] = acc;
    if (e2 != e) col2[i2] = acc2;
  }
}

// Entries a worker warp's lane updates while the pivot warp runs its chain
// (about 24 FP64 instructions, four to an entry).
constexpr int kChainEntries = 6;

// Takes the pivots [k0, k0 + kNb) (their eliminated columns: pan) to the next
// nb pivot columns and eliminates those; they are columns [l0, l0 + nb) of
// this CTA.  A warp per column first finishes its U rows and its rows of the
// pivot warp; while warp 0 then runs the chain of pivots (340 cycles each
// and 120 a further column), the warps of the
// other sub-partitions bring the remaining rows up to date, and with kRest
// (the front has one CTA) start on the columns [l0 + nb, l1) after them.
// Returns the entries of those already done.
template <class T, bool kRest>
__device__ __forceinline__ int next_block(T *F, int ld, int l0, int l1, int k0, int nb, int m, const T *pan, T *su,
                                          T *sr) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5, kn = k0 + kNb;
  T *base = F + size_t(l0) * ld;
  for (int c = w; c < nb; c += nw) {
    T *col = base + size_t(c) * ld;
    T u[kNb];
#pragma unroll
    for (int q = 0; q < kNb; ++q) u[q] = col[k0 + q];
#pragma unroll
    for (int q = 1; q < kNb; ++q)
#pragma unroll
      for (int s = 0; s < q; ++s) u[q] -= pan[s * ld + k0 + q] * u[s];
    __syncwarp();
    if (lane == 0) {
#pragma unroll
      for (int q = 1; q < kNb; ++q) col[k0 + q] = u[q];
    }
    const int i = kn + lane;
    if (i < m) {
      T acc = col[i];
#pragma unroll
      for (int q = 0; q < kNb; ++q) acc -= pan[q * ld + i] * u[q];
      col[i] = acc;
    }
  }
  __syncthreads();
  int done = 0;
  const int rem = m - kn, n_rest = kRest ? rem * (l1 - l0 - nb) : 0;
  if (w == 0) pivot_rows<T>(base, ld, kn, nb, m, su, sr);
  // the workers: every warp of sub-partitions 1 to 3, or the only warp
  const int workers = nw == 1 ? 1 : nw - (nw + 3) / 4, me = nw == 1 ? 0 : w - 1 - w / 4;
  if (nw == 1 || (w & 3)) {
    for (int i = kn + 32 + 32 * me + lane; i < m; i += 32 * workers) {
      T v[kNb];
#pragma unroll
      for (int s = 0; s < kNb; ++s) v[s] = s < nb ? base[size_t(s) * ld + i] : T(0);
#pragma unroll
      for (int q = 0; q < kNb; ++q) {
        const T l = pan[q * ld + i];
#pragma unroll
        for (int s = 0; s < kNb; ++s)
          if (s < nb) v[s] -= l * base[size_t(s) * ld + k0 + q];
      }
#pragma unroll
      for (int s = 0; s < kNb; ++s)
        if (s < nb) base[size_t(s) * ld + i] = v[s];
    }
  }
  if (kRest) {
    done = min(n_rest, nw == 1 ? n_rest : 32 * kChainEntries * workers);
    if (nw == 1 || (w & 3)) {
      update_u<T>(F, ld, l0 + nb, l1, pan, k0, kNb, 32 * me + lane, 32 * workers);
      if (nw == 1) __syncwarp();
      else asm volatile("bar.sync 1, %0;" ::"r"(32 * workers) : "memory");
      update_rest<T>(F, ld, l0 + nb, pan, k0, kNb, m, 0, done, 32 * me + lane, 32 * workers);
    }
  }
  __syncthreads();
  lower_rows<T>(base, ld, kn, nb, m, su, sr);
  return done;
}

// One CTA's part of a front, in W arithmetic; T is what is kept.
template <class W, class T>
__device__ void factor_front(const FrontDev &d, const Front f, const double *a, unsigned char *raw,
                             unsigned long long *bar, int limit) {
  const int C = f.ctas, r = C > 1 ? int(cluster_rank()) & (C - 1) : 0, rank0 = int(cluster_rank()) - r;
  const int m = f.m, p = f.p, ld = column_stride(m), tid = threadIdx.x, bd = blockDim.x;
  const int ncl = local_columns(m, r, C);
  W *su = reinterpret_cast<W *>(raw);       // pivot rows of the block being eliminated
  W *sr = su + kNb * kNb;                   // and their reciprocal pivots
  W *pb = sr + kNb;                         // another CTA's pivot columns
  W *F = pb + (C > 1 ? size_t(kNb) * ld : 0);
  assemble<W, T>(d, f, a, F, ld, ncl, r, C);
  __syncthreads();
  const int blocks = (p + kNb - 1) / kNb;
  if (C == 1) {
    if (tid < 32) pivot_rows<W>(F, ld, 0, min(kNb, p), m, su, sr);
    __syncthreads();
    lower_rows<W>(F, ld, 0, min(kNb, p), m, su, sr);
    __syncthreads();
    for (int jb = 0; jb < blocks; ++jb) {
      const int k0 = jb * kNb, nb = min(kNb, p - k0), nbn = min(kNb, p - k0 - kNb);
      const W *pan = F + size_t(k0) * ld;
      int l0 = k0 + nb, done = 0;
      if (jb + 1 < blocks) {
        done = next_block<W, true>(F, ld, l0, m, k0, nbn, m, pan, su, sr);
        l0 += nbn;
      } else {
        update_u<W>(F, ld, l0, m, pan, k0, nb, tid, bd);
        __syncthreads();
      }
      update_rest<W>(F, ld, l0, pan, k0, nb, m, done, (m - k0 - nb) * (m - l0), tid, bd);
      __syncthreads();
    }
  } else {
    // Block jb's columns are final in its owner's shared memory: a thread
    // tells each CTA of the front.  Barrier jb % C serves one block of each
    // round of C; a CTA owns one block of a round itself, so no barrier
    // completes twice before it is waited for.  In a wide front only the next
    // block's owner reads the columns there; it is told first, and the others
    // read them from the factor in L2 (15 readers of one SM's shared memory
    // took 2,400 cycles for 8 KB each, one takes 570).
    const bool wide = C > 4;
    auto hand_over = [&](int jb) {
      const int k0 = jb * kNb, nb = min(kNb, p - k0), next = jb + 1 < blocks ? (jb + 1) % C : -1;
      __syncthreads();
      if (!wide) {
        if (tid < C) signal(remote(bar + jb % C, unsigned(rank0 + tid)));
        return;
      }
      if (tid == 0 && next >= 0) signal(remote(bar + jb % C, unsigned(rank0 + next)));
      const W *src = F + size_t((jb / C) * kNb) * ld;
      T *dst = (T *)d.l + f.lo + int64_t(k0) * m;
      for (int i = k0 + tid; i < m; i += bd)
        for (int q = 0; q < nb; ++q) dst[int64_t(q) * m + i] = T(src[q * ld + i]);
      __syncthreads();
      if (tid < C && tid != next) signal(remote(bar + jb % C, unsigned(rank0 + tid)));
    };
    if (r == 0) {
      if (tid < 32) pivot_rows<W>(F, ld, 0, min(kNb, p), m, su, sr);
      __syncthreads();
      lower_rows<W>(F, ld, 0, min(kNb, p), m, su, sr);
      hand_over(0);
    }
    for (int jb = 0; jb < blocks; ++jb) {
      const int k0 = jb * kNb, nb = min(kNb, p - k0), own = jb % C, lc0 = (jb / C) * kNb;
      if (!await(smem_u32(bar + own), unsigned(jb / C) & 1u, limit)) atomicOr(d.status, 2u);
      const W *pan = F + size_t(lc0) * ld;
      // this CTA's first column after the block
      const int passed = jb >= r ? (jb - r) / C + 1 : 0;
      const bool next = jb + 1 < blocks && r == (jb + 1) % C;
      int l0 = r == own ? lc0 + nb : min(passed * kNb, ncl);
      if (r != own && l0 < ncl) {
        const int rows = m - k0, cnt = nb * rows;
        for (int e = tid; e < cnt; e += 4 * bd) {
          W *dst[4];
          W v[4];
          if (next || !wide) {
            unsigned src[4];
#pragma unroll
            for (int z = 0; z < 4; ++z) {
              const int ez = min(e + z * bd, cnt - 1), q = ez / rows, i = k0 + ez - q * rows;
              src[z] = remote(F + size_t(lc0 + q) * ld + i, unsigned(rank0 + own));
              dst[z] = pb + q * ld + i;
            }
            remote_load4(src, v);
          } else {
            const T *src = (const T *)d.l + f.lo + int64_t(k0) * m;
#pragma unroll
            for (int z = 0; z < 4; ++z) {
              const int ez = min(e + z * bd, cnt - 1), q = ez / rows, i = k0 + ez - q * rows;
              dst[z] = pb + q * ld + i;
              v[z] = W(__ldcg(src + int64_t(q) * m + i));
            }
          }
#pragma unroll
          for (int z = 0; z < 4; ++z) *dst[z] = v[z];  // past the end: the last entry again
        }
        pan = pb;
      }
      __syncthreads();
      if (next) {
        const int nbn = min(kNb, p - k0 - kNb);
        next_block<W, false>(F, ld, l0, ncl, k0, nbn, m, pan, su, sr);
        hand_over(jb + 1);
        l0 += nbn;
      }
      if (l0 < ncl) {
        update_u<W>(F, ld, l0, ncl, pan, k0, nb, tid, bd);
        __syncthreads();
        update_rest<W>(F, ld, l0, pan, k0, nb, m, 0, (m - k0 - nb) * (ncl - l0), tid, bd);
      }
      __syncthreads();
    }
  }
  // reciprocal pivots (here: a global store before a hand-over would have to
  // land first), factor and Schur complement, a warp per column
  for (int lc = tid; lc < ncl; lc += bd) {
    const int j = ((lc / kNb) * C + r) * kNb + lc % kNb;
    if (j < p) {
      const W pivot = F[size_t(lc) * ld + j];
      ((T *)d.rd)[f.pv + j] = T(pivot_reciprocal(pivot));
      if (bad_value(T(pivot))) report_pivot(d.status, __ldg(d.idx + f.idx + j));
    }
  }
  const int lane = tid & 31, b = m - p;
  for (int lc = tid >> 5; lc < ncl; lc += bd >> 5) {
    const int j = ((lc / kNb) * C + r) * kNb + lc % kNb;
    const W *col = F + size_t(lc) * ld;
    if (j < p) {
      // (a wide front's hand-over wrote the rows of the block and below)
      T *dst = (T *)d.l + f.lo + int64_t(j) * m;
      const int e = C > 4 ? j / kNb * kNb : m;
      for (int i = lane; i < e; i += 32) dst[i] = T(col[i]);
    } else {
      T *dst = (T *)d.u + f.uo + int64_t(j - p) * p;
      for (int i = lane; i < p; i += 32) dst[i] = T(col[i]);
      dst = (T *)d.c + f.co + int64_t(j - p) * b;
      for (int i = lane; i < b; i += 32) dst[i] = T(col[p + i]);
    }
  }
}

// slot: per CTA of the launch the front it works for (-1: none); a front's
// Front::ctas CTAs are neighbours in one cluster.
template <class T>
__global__ void __launch_bounds__(kFrontMax) front_factor(FrontDev d, const double *a, const int *__restrict__ slot,
                                                          const unsigned *limit_at) {
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ __align__(8) unsigned long long bar[kMaxCtas];
  const int number = __ldg(slot + blockIdx.x), tid = threadIdx.x;
  const bool shared_cluster = cluster_size() > 1;
  if (tid == 0) {
    for (int k = 0; k < kMaxCtas; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar + k)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (shared_cluster) cluster_sync();  // every barrier of the cluster is ready
  await_previous();
  if (number >= 0) {
    const Front f = d.front[number];
    const int limit = int(__ldg(limit_at));
    if (sizeof(T) == sizeof(double) || f.m <= kFrontDouble) factor_front<double, T>(d, f, a, raw, bar, limit);
    else factor_front<T, T>(d, f, a, raw, bar, limit);
  }
  if (shared_cluster) cluster_sync();  // no CTA leaves while another may read its columns
}

// Opens a refactor: keeps A for the rows outside the tree and refinement,
// resets the status.
__global__ void front_open(const double *a, double *a_copy, int64_t nnz, unsigned *status) {
  const int64_t t0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  await_previous();
  if (t0 == 0) {
    status[0] = 0;
    status[1] = 0xffffffffu;
  }
  if (a_copy != a)
    for (int64_t p = t0; p < nnz; p += int64_t(gridDim.x) * blockDim.x) a_copy[p] = a[p];
}

struct RowsDev {
  const int *row, *diag, *col, *a;
  const int64_t *ptr;
};

__global__ void front_check_rows(RowsDev R, int n, const double *a, unsigned *status) {
  await_previous();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (bad_value(a[R.diag[i]])) report_pivot(status, R.row[i]);
}

// One round of rows outside the tree (and the tree's right-hand sides, which
// have no pivot here): a cluster of kLongCtas blocks per long row first (a
// supply's row has an entry per device on it: 65 us with a block for each of
// 200,000 devices of logic's two), then a thread per row.  clear: flags the
// solve that follows starts from (nullptr: none).
constexpr int kLongCtas = 8, kLongThreads = 1024;
__global__ void __launch_bounds__(kLongThreads) front_rows(RowsDev R, int i0, int n_long, int n, const double *a,
                                                   const double *b, const int *__restrict__ P,
                                                   const int *__restrict__ Q, double *xk, double *x,
                                                   unsigned *clear, int n_clear) {
  __shared__ double part[32];
  const int bd = blockDim.x;
  // (a long row's blocks are one cluster, all of them; its barrier is waited
  // for behind the sums)
  const int block = int(blockIdx.x) - n_long * kLongCtas;
  const bool is_long = block < 0;
  if (is_long) cluster_arrive();
  await_previous();
  if (clear)
    for (int k = blockIdx.x * bd + threadIdx.x; k < n_clear; k += gridDim.x * bd) clear[k] = 0;
  const int i = is_long ? i0 + int(blockIdx.x) / kLongCtas : i0 + n_long + block * bd + int(threadIdx.x);
  if (i >= i0 + n) return;
  const int64_t e0 = R.ptr[i], e1 = R.ptr[i + 1];
  const int k = R.row[i], dg = R.diag[i];
  double s = 0.0;
  if (is_long) {
    __shared__ double sums[kLongCtas];
    const int rank = int(cluster_rank());
#pragma unroll 8
    for (int64_t e = e0 + rank * bd + threadIdx.x; e < e1; e += kLongCtas * bd) s += a[R.a[e]] * xk[R.col[e]];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    cluster_wait();  // every block of the row has started
    __syncthreads();
    if (threadIdx.x == 0) {
      s = part[0];
      for (int w = 1; w < bd >> 5; ++w) s += part[w];
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote(sums + rank, 0u)), "d"(s) : "memory");
    }
    cluster_sync();
    if (rank || threadIdx.x) return;
    s = sums[0];
    for (int w = 1; w < kLongCtas; ++w) s += sums[w];
  } else {
    for (int64_t e = e0; e < e1; ++e) s += a[R.a[e]] * xk[R.col[e]];
  }
  double v = b[P[k]] - s;
  if (dg >= 0) {
    v /= a[dg];
    x[Q[k]] = v;
  }
  xk[k] = v;
}

// The children's border sums that row i of a front gathers, in their order.
// Four children's places are found ahead of the wait for them, and their
// loads are in flight together.
constexpr int kAhead = 4;
__device__ __forceinline__ void find_children(const FrontDev &d, const Front &f, int c0, int i, int64_t (&at)[kAhead]) {
#pragma unroll
  for (int q = 0; q < kAhead; ++q) {
    at[q] = -1;
    if (c0 + q < f.child1) {
      const ChildDev &g = d.child[c0 + q];
      const int k = __ldg(d.inv_map + g.inv + i);
      if (k >= 0) at[q] = g.bv + k;
    }
  }
}
template <class T>
__device__ __forceinline__ T add_children(const FrontDev &d, T s, const int64_t (&at)[kAhead]) {
  T v[kAhead];
#pragma unroll
  for (int q = 0; q < kAhead; ++q) v[q] = at[q] >= 0 ? __ldcg((const T *)d.bv + at[q]) : T(0);
#pragma unroll
  for (int q = 0; q < kAhead; ++q) s += v[q];
  return s;
}

// The solves of a front go 32 pivots at a time.  Warp 0 resolves a block lane
// to lane (a pivot costs a shuffle and one FP64 instruction, 95 cycles); all
// warps then bring the next 32 rows up to date, and the rows beyond them
// follow while warp 0 resolves the next block.
//
// A block of fewer than 32 columns goes by eights, the last of them repeating
// its last column with a factor of 0: loads under a condition each would go
// one by one (up to 32 L2 round trips, 11 us a block).
//
// A lane's row of a block of pivots: its entries in the block's other columns
// that are solved before it (below the diagonal forward, above it backward).
template <class T, bool kUp>
__device__ __forceinline__ void load_block(const T *L, int m, int kb, int nb, T (&w)[32]) {
  const int lane = threadIdx.x & 31;
  const T *col = L + int64_t(kb) * m + kb + min(lane, nb - 1);
#pragma unroll
  for (int g = 0; g < 32; g += 8)
    if (g < nb)
#pragma unroll
      for (int t = g; t < g + 8; ++t) w[t] = col[int64_t(min(t, nb - 1)) * m];
#pragma unroll
  for (int t = 0; t < 32; ++t) w[t] = t < nb && lane < nb && (kUp ? lane > t : lane < t) ? w[t] : T(0);
}
// v less the columns [kb, kb + nb) in the rows [i0, i1): a row per thread (t
// of n), ...
template <class T>
__device__ __forceinline__ void apply_rows(const T *L, int m, T *v, int kb, int nb, int i0, int i1, int t, int n) {
  for (int i = i0 + t; i < i1; i += n) {
    T w[32], s = v[i];
    if (nb == 32) {
#pragma unroll
      for (int q = 0; q < 32; ++q) w[q] = L[int64_t(kb + q) * m + i];
#pragma unroll
      for (int q = 0; q < 32; ++q) s -= w[q] * v[kb + q];
    } else {
      for (int g = 0; g < nb; g += 8) {
#pragma unroll
        for (int q = 0; q < 8; ++q) w[q] = L[int64_t(kb + min(g + q, nb - 1)) * m + i];
#pragma unroll
        for (int q = 0; q < 8; ++q) s -= (g + q < nb ? w[q] : T(0)) * v[kb + min(g + q, nb - 1)];
      }
    }
    v[i] = s;
  }
}
// ... and in the 32 rows from i0 on: 8 rows to a warp, 8 columns to a lane.
template <class T>
__device__ __forceinline__ void apply_next(const T *L, int m, T *v, int kb, int nb, int i0, int i1) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, c0 = (lane >> 3) * 8;
  for (int g = threadIdx.x >> 5; g < 4; g += nw) {
    const int i = i0 + 8 * g + (lane & 7), row = min(i, i1 - 1);
    T w[8], s = T(0);
#pragma unroll
    for (int q = 0; q < 8; ++q) w[q] = L[int64_t(kb + min(c0 + q, nb - 1)) * m + row];
#pragma unroll
    for (int q = 0; q < 8; ++q) s += (c0 + q < nb ? w[q] : T(0)) * v[kb + min(c0 + q, nb - 1)];
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 16);
    if (lane < 8 && i < i1) v[i] -= s;
  }
}

// y = L \\ (right-hand side and the children's sums) for the front's pivots;
// its border sums go to its parent.  What does not depend on other fronts is
// loaded ahead: warp 0's first block, the other warps' row of it where it is
// the only one, the places of the children's sums, the right-hand side.
template <class T>
struct Up {
  T w[32], rhs;
  int64_t at[kAhead];
};
template <class T>
__device__ __forceinline__ void ahead(const FrontDev &d, const Front &f, Up<T> &a) {
  const int m = f.m, p = f.p, tid = threadIdx.x, nb = min(32, p), i = nb + tid - 32;
  const T *L = (const T *)d.l + f.lo;
  if (tid < 32) {
    load_block<T, true>(L, m, 0, nb, a.w);
  } else if (p <= 32) {
#pragma unroll
    for (int g = 0; g < 32; g += 8)
      if (g < nb)
#pragma unroll
        for (int q = g; q < g + 8; ++q) a.w[q] = L[int64_t(min(q, nb - 1)) * m + min(i, m - 1)];
  }
  a.rhs = tid < p ? T(__ldcg(d.xk + __ldg(d.idx + f.idx + tid))) : T(0);
  if (tid < m) find_children(d, f, f.child0, tid, a.at);
}
template <class T>
__device__ __forceinline__ void forward(const FrontDev &d, const Front &f, T *v, Up<T> &a) {
  const int m = f.m, p = f.p, tid = threadIdx.x, bd = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = bd >> 5;
  const T *L = (const T *)d.l + f.lo;
  for (int i = tid; i < m; i += bd) {
    T r = a.rhs;
    if (i != tid) {
      r = i < p ? T(__ldcg(d.xk + __ldg(d.idx + f.idx + i))) : T(0);
      find_children(d, f, f.child0, i, a.at);
    }
    T s = add_children<T>(d, T(0), a.at);
    for (int c = f.child0 + kAhead; c < f.child1; c += kAhead) {
      find_children(d, f, c, i, a.at);
      s = add_children<T>(d, s, a.at);
    }
    v[i] = s + r;
  }
  __syncthreads();
  for (int kb = 0; kb < p; kb += 32) {
    const int nb = min(32, p - kb);
    if (wid == 0) {
      T s = lane < nb ? v[kb + lane] : T(0);
#pragma unroll
      for (int t = 0; t < 32; ++t) {
        if (t < nb) {
          const T vt = __shfl_sync(0xffffffffu, s, t), r = s - a.w[t] * vt;
          s = lane > t ? r : s;
        }
      }
      if (lane < nb) {
        v[kb + lane] = s;
        ((T *)d.y)[f.pv + kb + lane] = s;
      }
    }
    if (kb > 0 && (wid > 0 || nw == 1))
      apply_rows<T>(L, m, v, kb - 32, 32, kb + 32, m, nw == 1 ? tid : tid - 32, nw == 1 ? bd : bd - 32);
    __syncthreads();
    if (kb + 32 < p) {
      if (wid == 0) load_block<T, true>(L, m, kb + 32, min(32, p - kb - 32), a.w);
      apply_next<T>(L, m, v, kb, 32, kb + 32, m);
    } else if (p <= 32 && nw > 1) {
      const int i = nb + tid - 32;
      if (wid > 0 && i < m) {
        T s = v[i];
#pragma unroll
        for (int q = 0; q < 32; ++q)
          if (q < nb) s -= a.w[q] * v[q];
        v[i] = s;
      }
      apply_rows<T>(L, m, v, 0, nb, nb + bd - 32, m, tid, bd);
    } else {
      apply_rows<T>(L, m, v, kb, nb, kb + nb, m, tid, bd);
    }
    __syncthreads();
  }
  for (int i = p + tid; i < m; i += bd) ((T *)d.bv)[f.bv + i - p] = v[i];
}

// x = U \\ (y - the border's part) for the front's pivots, border first; v
// holds m values and p per warp.  Ahead: warp 0's last block, the first of a
// warp's columns of U, the border's unknowns' places.
constexpr int kAheadU = 8;
template <class T>
struct Down {
  T w[32], u[kAheadU], rd;
  int at, own, own_x;
};
template <class T>
__device__ __forceinline__ void ahead(const FrontDev &d, const Front &f, Down<T> &a) {
  const int m = f.m, p = f.p, b = m - p, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
  const int kb = (p - 1) / 32 * 32;
  const T *U = (const T *)d.u + f.uo;
  if (tid < 32) load_block<T, false>((const T *)d.l + f.lo, m, kb, p - kb, a.w);
  a.rd = tid < p - kb ? ((const T *)d.rd)[f.pv + kb + tid] : T(0);
#pragma unroll
  for (int q = 0; q < kAheadU; ++q) {
    const int j = wid + q * nw;
    if (b > 0) a.u[q] = U[int64_t(min(j, b - 1)) * p + min(lane, p - 1)];
  }
  a.at = tid < b ? __ldg(d.idx + f.idx + p + tid) : 0;
  a.own = tid < p ? __ldg(d.idx + f.idx + tid) : 0;
  a.own_x = tid < p ? __ldg(d.Q + a.own) : 0;
}
template <class T>
__device__ __forceinline__ void backward(const FrontDev &d, const Front &f, T *v, Down<T> &a, double *x) {
  const int m = f.m, p = f.p, b = m - p, tid = threadIdx.x, bd = blockDim.x, lane = tid & 31;
  const int wid = tid >> 5, nw = bd >> 5;
  T *xb = v + p;                      // the border's unknowns
  T *red = xb + b;                    // the warps' sums
  const T *L = (const T *)d.l + f.lo, *U = (const T *)d.u + f.uo;
  for (int j = tid; j < b; j += bd) xb[j] = T(__ldcg(d.xk + (j == tid ? a.at : __ldg(d.idx + f.idx + p + j))));
  for (int i = tid; i < p; i += bd) v[i] = __ldcg((const T *)d.y + f.pv + i);
  __syncthreads();
  // v = y - U x: every warp a share of the border for all rows, the shares
  // added in order
  for (int i = lane; i < p; i += 32) {
    T s = T(0);
    int j = wid;
    if (i == lane) {
#pragma unroll
      for (int q = 0; q < kAheadU; ++q, j += nw)
        if (j < b) s += a.u[q] * xb[j];
    }
#pragma unroll 16
    for (; j < b; j += nw) s += U[int64_t(j) * p + i] * xb[j];
    red[wid * p + i] = s;
  }
  __syncthreads();
  for (int i = tid; i < p; i += bd) {
    T t = v[i];
    for (int q = 0; q < nw; ++q) t -= red[q * p + i];
    v[i] = t;
  }
  __syncthreads();
  for (int kb = ((p - 1) / 32) * 32; kb >= 0; kb -= 32) {
    const int nb = min(32, p - kb);
    if (wid == 0) {
      T s = lane < nb ? v[kb + lane] : T(0);
#pragma unroll
      for (int t = 31; t >= 0; --t) {
        if (t < nb) {
          const T vt = __shfl_sync(0xffffffffu, s, t) * __shfl_sync(0xffffffffu, a.rd, t);
          const T r = s - a.w[t] * vt;
          s = lane == t ? vt : lane < t ? r : s;
        }
      }
      if (lane < nb) v[kb + lane] = s;
    }
    if (kb + 32 < p && (wid > 0 || nw == 1))
      apply_rows<T>(L, m, v, kb + 32, min(32, p - kb - 32), 0, kb, nw == 1 ? tid : tid - 32,
                    nw == 1 ? bd : bd - 32);
    __syncthreads();
    if (kb > 0) {
      if (wid == 0) {
        load_block<T, false>(L, m, kb - 32, 32, a.w);
        a.rd = ((const T *)d.rd)[f.pv + kb - 32 + lane];
      }
      apply_next<T>(L, m, v, kb, nb, kb - 32, kb);
      __syncthreads();
    }
  }
  for (int i = tid; i < p; i += bd) {
    const int k = i == tid ? a.own : __ldg(d.idx + f.idx + i);
    d.xk[k] = double(v[i]);
    x[i == tid ? a.own_x : __ldg(d.Q + k)] = double(v[i]);
  }
}

template <class T>
__global__ void __launch_bounds__(256) front_forward(FrontDev d, int f0) {
  extern __shared__ __align__(16) unsigned char raw[];
  const Front f = d.front[f0 + blockIdx.x];
  await_previous();
  Up<T> a;
  ahead<T>(d, f, a);
  forward<T>(d, f, reinterpret_cast<T *>(raw), a);
}
template <class T>
__global__ void __launch_bounds__(256) front_backward(FrontDev d, int f0, double *x) {
  extern __shared__ __align__(16) unsigned char raw[];
  const Front f = d.front[f0 + blockIdx.x];
  await_previous();
  Down<T> a;
  ahead<T>(d, f, a);
  backward<T>(d, f, reinterpret_cast<T *>(raw), a, x);
}

// Polls a flag (acquire) until it is set, at most `limit` times.
__device__ __forceinline__ bool wait_flag(const unsigned *p, int limit) {
  unsigned v = 0;
  for (int it = 0; it < limit; ++it) {
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    if (v) return true;
    if (it > 32) __nanosleep(32);
  }
  return false;
}

// Both solves over the fronts above level 0 in one launch.  Blocks claim
// fronts in order, children before parents, then in reverse; a front waits
// (bounded) for its children's border sums, backward for its parent, so a
// step up or down the tree costs a flag and the front's own work instead of
// a launch that waits for the whole level.  Every front waited for was
// claimed earlier by a running block, so the claims always advance.  What
// bounds it is the tree's height: per front the wait, the children's sums,
// the pivots' chain and the flag, with everything static loaded before the
// wait (a 28-pivot front 3.6 us up, 8.9 with its loads after it).  Measured:
// 60x60 power grid 113 us (141), 200x200 361 (440), 200,000 devices of logic
// 448 (512).  flow:
// the claim counter, then a forward and a backward flag per front, cleared
// before the launch.
template <class T, int kPerSm>
__global__ void __launch_bounds__(kFlowThreads, kPerSm) front_flow(FrontDev d, int first, int nf, unsigned *flow,
                                                           const unsigned *limit_at, double *x) {
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ int claim;
  const int count = nf - first, limit = int(__ldg(limit_at)), tid = threadIdx.x;
  unsigned *fwd = flow + 1, *bwd = fwd + nf;
  await_previous();
  for (;;) {
    if (tid == 0) claim = int(atomicAdd(flow, 1u));
    __syncthreads();
    const int t = claim;
    if (t >= 2 * count) break;
    const bool up = t < count;
    const int k = up ? first + t : nf - 1 - (t - count);
    const Front f = d.front[k];
    if (up) {
      Up<T> a;
      ahead<T>(d, f, a);
      bool ok = true;
      for (int c = f.child0 + tid; c < f.child1; c += kFlowThreads) {
        const int g = d.child[c].front;
        if (g >= first) ok = wait_flag(fwd + g, limit) && ok;
      }
      if (!ok) atomicOr(d.status, 2u);
      __syncthreads();
      forward<T>(d, f, reinterpret_cast<T *>(raw), a);
    } else {
      Down<T> a;
      ahead<T>(d, f, a);
      if (tid == 0 && !wait_flag(f.parent >= 0 ? bwd + f.parent : fwd + k, limit)) atomicOr(d.status, 2u);
      __syncthreads();
      backward<T>(d, f, reinterpret_cast<T *>(raw), a, x);
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"((up ? fwd : bwd) + k), "r"(1u) : "memory");
    }
  }
}

// The largest |multiplier| per front.
template <class T>
__global__ void __launch_bounds__(256) front_multipliers(FrontDev d, double *out) {
  __shared__ double part[8];
  const Front f = d.front[blockIdx.x];
  const T *L = (const T *)d.l + f.lo;
  double mx = 0.0;
  for (int64_t e = threadIdx.x; e < int64_t(f.m) * f.p; e += 256) {
    const int64_t j = e / f.m;
    if (e - j * f.m > j) {
      const double v = fabs(double(L[e]));
      mx = v > mx || v != v ? v : mx;  // a NaN stays
    }
  }
  // NaN-keeping maximum over the block
  for (int o = 16; o > 0; o >>= 1) {
    const double v = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = v > mx || v != v ? v : mx;
  }
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) mx = part[w] > mx || part[w] != part[w] ? part[w] : mx;
    out[blockIdx.x] = mx;
  }
}

struct Group {  // fronts of one level launched together
  int f0, n;                      // solves of level 0
  int slot0, grid, cluster, threads;
  size_t smem, smem_fwd, smem_bwd;
  int solve_threads;
};

}  // namespace

struct FrontLu {
  int n = 0, n_front = 0;
  int precision = 0;
  std::vector<Group> group;
  std::vector<void *> owned;
  FrontDev d{};
  RowsDev before{}, core{}, after{};
  std::vector<int> before_round, core_round, after_round;
  bool flow_many = false;
  int flow_first = 0, flow_grid = 0;  // fronts from here on (levels above 0) are solved in one launch
  size_t n_low = 0;                   // groups of level 0
  size_t flow_smem = 0;
  unsigned *flow = nullptr;           // claim counter and flags
  const int *slot = nullptr;          // the factor launches' CTAs: their fronts
  ~FrontLu() {
    for (void *p : owned) cudaFree(p);
  }
};

namespace {

// One allocation that the LU owns.
template <class V>
bool take(FrontLu *f, V **p, size_t count) {
  *p = nullptr;
  if (cudaMalloc((void **)p, sizeof(V) * std::max<size_t>(count, 1)) != cudaSuccess) return false;
  f->owned.push_back(*p);
  return true;
}
template <class V>
bool give(FrontLu *f, const V **p, const std::vector<V> &src) {
  V *q = nullptr;
  if (!take(f, &q, src.size())) return false;
  *p = q;
  return src.empty() ||
         cudaMemcpy(q, src.data(), sizeof(V) * src.size(), cudaMemcpyHostToDevice) == cudaSuccess;
}
bool give_rows(FrontLu *f, RowsDev *R, const FrontRows &H) {
  return give(f, &R->row, H.row) && give(f, &R->diag, H.diag) && give(f, &R->col, H.col) && give(f, &R->a, H.a) &&
         give(f, &R->ptr, H.ptr);
}

// Whether the device can run clusters of so many such blocks at all (a
// partition of it may hold fewer SMs a cluster than the whole).
bool granted(const void *fn, int cluster, int threads, size_t smem) {
  if (cluster <= 1) return true;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(cluster));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = unsigned(cluster);
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int clusters = 0;
  return cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) == cudaSuccess && clusters > 0;
}

template <class T>
const void *factor_fn() {
  return (const void *)front_factor<T>;
}

// Fronts per SM from which the solves' walk takes four blocks an SM, with
// fewer registers, instead of two: it is then bound by how many fronts are in
// flight, not by one front's time (200,000 devices of logic, 4,946 fronts: 439
// us against 498; a 200x200 grid, 2,172 fronts: 402 against 394).
constexpr int kManyFronts = 16;
constexpr double kWideWork = 6e4;  // multiply-adds one SM is left with

}  // namespace

FrontLu *front_create(const FrontPlan &plan, const LuSymbolic &S, int device, int precision) {
  std::unique_ptr<FrontLu> f(new FrontLu);
  f->n = plan.n;
  f->n_front = int(plan.front.size());
  f->precision = precision;
  const size_t tsz = precision == XG_LU_FP32 ? sizeof(float) : sizeof(double);
  const void *fn = precision == XG_LU_FP32 ? factor_fn<float>() : factor_fn<double>();
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  std::vector<Front> front = plan.front;
  std::vector<int> slot;
  size_t most = 0;
  for (size_t l = 0; l + 1 < plan.level.size(); ++l) {
    const int at = plan.level[l], end = plan.level[l + 1];
    // the small fronts of a level with many apart: their blocks are smaller
    int first_small = at, first_low = at;
    while (first_small < end && plan.front[first_small].m > kFrontMiddle) ++first_small;
    while (first_low < end && plan.front[first_low].m > kFrontLow) ++first_low;
    std::vector<int> cut = {at};
    if (first_small > at && end - first_small > sms) cut.push_back(first_small);
    if (first_low > cut.back() && end - first_low > 4 * sms) cut.push_back(first_low);
    cut.push_back(end);
    for (size_t q = 0; q + 1 < cut.size(); ++q) {
      Group g{};
      g.f0 = cut[q];
      g.n = cut[q + 1] - cut[q];
      int m = 0;
      double total = 0.0;
      for (int k = g.f0; k < g.f0 + g.n; ++k) {
        m = std::max(m, front[k].m);
        total += front_work(front[k].p, front[k].m);
      }
      g.threads = std::max(m <= kFrontLow && g.n > 4 * sms ? 32 : 128, (m + 31) / 32 * 32);
      g.solve_threads = m <= kFrontLow ? 32 : m <= kFrontMiddle ? 64 : 256;
      // CTAs of a front: what brings its work down to an SM's share of the
      // level (below kWideWork another halving gains less than its
      // hand-overs cost) and its shared memory to a quarter of an SM's, so
      // that fronts hide each other's waits; at least two column blocks each
      const double share = std::max(kWideWork, total / sms);
      std::vector<int> by_ctas[5];
      for (int k = g.f0; k < g.f0 + g.n; ++k) {
        Front &h = front[k];
        int lg = 0;
        const double w = front_work(h.p, h.m);
        while (lg < 4 && (w > share * (1 << lg) || factor_smem(h.m, 1 << lg, tsz) > kSmemTarget) &&
               (4 * kNb << lg) <= h.m)
          ++lg;
        while (lg < 4 && factor_smem(h.m, 1 << lg, tsz) > kSmemLimit) ++lg;
        if (factor_smem(h.m, 1 << lg, tsz) > kSmemLimit) return nullptr;
        h.ctas = 1 << lg;
        by_ctas[lg].push_back(k);
        g.smem = std::max(g.smem, factor_smem(h.m, h.ctas, tsz));
      }
      // widest first: powers of two pack the clusters without gaps
      g.slot0 = int(slot.size());
      g.cluster = 1;
      for (int lg = 4; lg >= 0; --lg)
        for (int k : by_ctas[lg]) {
          g.cluster = std::max(g.cluster, 1 << lg);
          slot.insert(slot.end(), size_t(1) << lg, k);
        }
      while ((slot.size() - size_t(g.slot0)) % size_t(g.cluster)) slot.push_back(-1);
      g.grid = int(slot.size()) - g.slot0;
      g.smem_fwd = size_t(m) * tsz;
      int most_p = 0;
      for (int k = g.f0; k < g.f0 + g.n; ++k) most_p = std::max(most_p, front[k].p);
      g.smem_bwd = (size_t(m) + size_t(g.solve_threads / 32) * size_t(most_p)) * tsz;
      most = std::max(most, g.smem);
      f->group.push_back(g);
    }
    if (l == 0) f->n_low = f->group.size();
  }
  f->flow_first = plan.level.size() > 1 ? plan.level[1] : f->n_front;
  {
    size_t mx = 0;
    for (int k = f->flow_first; k < f->n_front; ++k)
      mx = std::max(mx, size_t(plan.front[k].m) + size_t(kFlowThreads / 32) * size_t(plan.front[k].p));
    f->flow_smem = mx * tsz;
    f->flow_many = f->n_front - f->flow_first > kManyFronts * sms;
    const void *flow_fn = precision == XG_LU_FP32
                              ? f->flow_many ? (const void *)front_flow<float, 4> : (const void *)front_flow<float, 2>
                          : f->flow_many ? (const void *)front_flow<double, 4>
                                         : (const void *)front_flow<double, 2>;
    int occ = 0;
    if (allow_dynamic_smem(flow_fn, f->flow_smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, flow_fn, kFlowThreads, f->flow_smem) != cudaSuccess)
      return nullptr;
    f->flow_grid = std::max(1, std::min(sms * std::max(occ, 1), f->n_front - f->flow_first));
  }
  if (allow_dynamic_smem(fn, most) != cudaSuccess) return nullptr;
  for (const Group &g : f->group)
    if (!granted(fn, g.cluster, g.threads, g.smem)) return nullptr;
  for (const FrontRows *R : {&plan.before, &plan.core, &plan.after})
    for (size_t k = 0; k + 2 < R->round.size(); k += 2)
      if (R->round[k + 1] > R->round[k] && !granted((const void *)front_rows, kLongCtas, kLongThreads, 0)) return nullptr;
  std::vector<ChildDev> child(plan.child.size());
  std::vector<int> own(plan.map.size(), 0), own_at;
  for (const Front &h : front)
    for (int k = h.child0; k < h.child1; ++k) {
      const Front &g = plan.front[plan.child[size_t(k)]];
      const int b = g.m - g.p, *map = plan.map.data() + g.map;
      child[size_t(k)] = ChildDev{plan.inv[size_t(k)], g.co, g.bv, g.map, b, plan.child[size_t(k)], int(own_at.size())};
      std::vector<int> count(size_t(h.ctas) + 1, 0);
      for (int j = 0; j < b; ++j) ++count[size_t(map[j] / kNb % h.ctas) + 1];
      for (int r = 0; r < h.ctas; ++r) count[size_t(r) + 1] += count[size_t(r)];
      own_at.insert(own_at.end(), count.begin(), count.end());
      for (int j = 0; j < b; ++j)
        own[size_t(g.map) + size_t(count[size_t(map[j] / kNb % h.ctas)]++)] =
            j | (map[j] / kNb / h.ctas * kNb + map[j] % kNb) << 16;
    }
  FrontDev &d = f->d;
  unsigned char *l = nullptr, *u = nullptr, *c = nullptr, *rd = nullptr, *y = nullptr, *bv = nullptr;
  const bool ok = give(f.get(), &d.front, front) && give(f.get(), &f->slot, slot) && give(f.get(), (const ChildDev **)&d.child, child) &&
                  give(f.get(), &d.idx, plan.idx) && give(f.get(), &d.map, plan.map) &&
                  give(f.get(), &d.inv_map, plan.inv_map) && give(f.get(), &d.own, own) &&
                  give(f.get(), &d.own_at, own_at) && give(f.get(), &d.apos, plan.apos) &&
                  give(f.get(), &d.aidx, plan.aidx) &&
                  give(f.get(), &d.P, S.P) && give(f.get(), &d.Q, plan.Q) && take(f.get(), &l, tsz * plan.n_l) &&
                  take(f.get(), &u, tsz * plan.n_u) && take(f.get(), &c, tsz * plan.n_c) &&
                  take(f.get(), &rd, tsz * plan.n_pv) && take(f.get(), &y, tsz * plan.n_pv) &&
                  take(f.get(), &bv, tsz * plan.n_bv) &&
                  take(f.get(), &f->flow, size_t(2 * f->n_front + 1)) && take(f.get(), &d.xk, size_t(plan.n)) &&
                  give_rows(f.get(), &f->before, plan.before) && give_rows(f.get(), &f->core, plan.core) &&
                  give_rows(f.get(), &f->after, plan.after);
  if (!ok) return nullptr;
  d.l = l;
  d.u = u;
  d.c = c;
  d.rd = rd;
  d.y = y;
  d.bv = bv;
  f->before_round = plan.before.round;
  f->core_round = plan.core.round;
  f->after_round = plan.after.round;
  return f.release();
}

void front_destroy(FrontLu *f) { delete f; }

int front_refactor(FrontLu *f, const double *dev_values, double *a_copy, int64_t nnz_a, unsigned *status,
                   const unsigned *limit, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  f->d.status = status;
  cudaError_t e = launch_close(front_open, int(std::min<int64_t>(1024, (nnz_a + 255) / 256)), 256, 0, 0, s, dev_values,
                         a_copy, nnz_a, status);
  for (const Group &g : f->group) {
    if (e != cudaSuccess) return XG_ERR_CUDA;
    e = launch_close(f->precision == XG_LU_FP32 ? front_factor<float> : front_factor<double>, g.grid, g.threads, g.smem,
               g.cluster, s, f->d, dev_values, f->slot + g.slot0, limit);
  }
  const RowsDev *rows[] = {&f->before, &f->after};
  const std::vector<int> *round[] = {&f->before_round, &f->after_round};
  for (int k = 0; k < 2; ++k) {
    if (round[k]->empty() || !round[k]->back()) continue;
    const int n = round[k]->back();
    if (e == cudaSuccess)
      e = launch_close(front_check_rows, std::min(1024, (n + 255) / 256), 256, 0, 0, s, *rows[k], n, a_copy, status);
  }
  return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? XG_OK : XG_ERR_CUDA;
}

template <class T>
static cudaError_t solve_tree(FrontLu *f, double *x, unsigned *status, const unsigned *limit, cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  for (size_t k = 0; k < f->n_low && e == cudaSuccess; ++k) {
    const Group &g = f->group[k];
    e = launch_close(front_forward<T>, g.n, g.solve_threads, g.smem_fwd, 0, s, f->d, g.f0);
  }
  if (f->flow_first < f->n_front && e == cudaSuccess) {
    f->d.status = status;
    e = launch_close(f->flow_many ? front_flow<T, 4> : front_flow<T, 2>, f->flow_grid, kFlowThreads, f->flow_smem, 0, s, f->d,
               f->flow_first, f->n_front, f->flow, limit, x);
  }
  for (size_t k = f->n_low; k-- > 0 && e == cudaSuccess;) {
    const Group &g = f->group[k];
    e = launch_close(front_backward<T>, g.n, g.solve_threads, g.smem_bwd, 0, s, f->d, g.f0, x);
  }
  return e;
}

int front_solve(FrontLu *f, const double *a_copy, const double *b, double *x, unsigned *status, const unsigned *limit,
                void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaSuccess;
  auto rows = [&](const RowsDev &R, const std::vector<int> &round, unsigned *clear) {
    for (size_t k = 0; k + 2 < round.size() && e == cudaSuccess; k += 2) {
      const int i0 = round[k], n_long = round[k + 1] - i0, n = round[k + 2] - i0;
      if (!n) continue;
      const int bd = n_long ? kLongThreads : 256, short_blocks = (n - n_long + bd - 1) / bd;
      const int grid = n_long ? n_long * kLongCtas + (short_blocks + kLongCtas - 1) / kLongCtas * kLongCtas : short_blocks;
      e = launch_close(front_rows, grid, bd, 0, n_long ? kLongCtas : 0, s, R, i0, n_long, n, a_copy, b, f->d.P, f->d.Q,
                 f->d.xk, x, clear, 2 * f->n_front + 1);
    }
  };
  rows(f->before, f->before_round, nullptr);
  rows(f->core, f->core_round, f->flow);
  if (e == cudaSuccess)
    e = f->precision == XG_LU_FP32 ? solve_tree<float>(f, x, status, limit, s)
                                   : solve_tree<double>(f, x, status, limit, s);
  rows(f->after, f->after_round, nullptr);
  return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? XG_OK : XG_ERR_CUDA;
}

int front_max_multiplier(FrontLu *f, double *out, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  double *dev = nullptr;
  std::vector<double> h(size_t(f->n_front), 0.0);
  if (cudaMalloc((void **)&dev, sizeof(double) * h.size()) != cudaSuccess) return XG_ERR_OOM;
  if (f->precision == XG_LU_FP32) front_multipliers<float><<<f->n_front, 256, 0, s>>>(f->d, dev);
  else front_multipliers<double><<<f->n_front, 256, 0, s>>>(f->d, dev);
  count_launches(1);
  cudaError_t e = cudaMemcpyAsync(h.data(), dev, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, s);
  const cudaError_t e2 = cudaStreamSynchronize(s);
  cudaFree(dev);
  if (e != cudaSuccess || e2 != cudaSuccess) return XG_ERR_CUDA;
  double mx = 0.0;
  for (double v : h) mx = v > mx || v != v ? v : mx;
  *out = mx;
  return XG_OK;
}

}  // namespace xg
