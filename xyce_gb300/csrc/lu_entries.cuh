// lu_entries.cuh — a small factor in shared memory, entry by entry (device
// side of LuEntries, xg_lu.h).
//
// The schedule orders the entries of L\U by when their inputs are final: an
// entry pulls all its updates at once (val -= l u per pair, in the
// elimination's order) and is then scaled by its reciprocal pivot (L), left
// (U), or becomes a pivot.  Entries of one level are independent; a thread
// takes each, a warp those with many pairs.  A row of the forward solve takes
// part as soon as its L entries and the values they meet are final, so a
// refactor with a solve needs no forward levels of its own.  On GB300 an FP64
// instruction costs a sub-partition 66 cycles and a shared-memory load 37: a
// thread per row spent most of a level following the row's index chain
// (4,000 cycles a level on a 1,000-stage inverter chain, 85,000 in all, its
// supply row another 36,000).
#pragma once

#include <cuda_runtime.h>

#include "xg_fast_rcp.cuh"
#include "xg_lu.h"

namespace xg {

// 1 / u: a Halley step (the cubic member of Householder's family: with
// e = 1 - u x, x (1 + e + e^2) leaves a relative error of e^3) from the
// hardware's 20-bit approximation, three multiply-adds where the IEEE
// division has a longer chain; pivots follow one another at its latency.
// The division itself near the ends of the exponent range.
__device__ __forceinline__ double pivot_reciprocal(double u) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(u));
  const double e = fma(-u, x, 1.0);
  x = fma(x, fma(e, e, e), x);
  const int ex = (__double2hiint(u) >> 20) & 0x7ff;
  if (unsigned(ex - 64) > 1918u) x = 1.0 / kept_apart(u);
  return x;
}
__device__ __forceinline__ float pivot_reciprocal(float u) { return 1.0f / u; }

// A zero, infinite or NaN pivot, from the bits (no FP64 instruction).
__device__ __forceinline__ bool bad_value(double u) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(u);
  return (b << 1) == 0 || ((b >> 52) & 0x7ff) == 0x7ff;
}
__device__ __forceinline__ bool bad_value(float u) {
  const unsigned b = __float_as_uint(u);
  return (b << 1) == 0 || ((b >> 23) & 0xff) == 0xff;
}

template <class T>
__device__ __forceinline__ T butterfly_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The factor in shared memory and its schedule: img[w] is word w of the image
// (only the words of the parts that were staged are there).
template <class T>
struct EntryView {
  T *val, *rd, *y;
  const uint32_t *img;
  LuEntriesHead h;

  __device__ const uint16_t *u16(int word) const { return reinterpret_cast<const uint16_t *>(img + word); }
  __device__ const uint16_t *ci() const { return u16(h.ci); }
  __device__ const uint16_t *rp() const { return u16(h.rp); }
  __device__ const uint16_t *diag() const { return u16(h.diag); }
};

// y[i] less its L part: serially, or by a warp for a long row.
template <class T>
__device__ __forceinline__ void forward_row(const EntryView<T> &v, int i) {
  const uint16_t *ci = v.ci();
  T acc = v.y[i];
  int p = v.rp()[i];
  const int e = v.diag()[i];
  for (; p + 4 <= e; p += 4) {  // (loads ahead of their multiply-adds)
    const int k0 = ci[p], k1 = ci[p + 1], k2 = ci[p + 2], k3 = ci[p + 3];
    const T a0 = v.val[p], a1 = v.val[p + 1], a2 = v.val[p + 2], a3 = v.val[p + 3];
    const T y0 = v.y[k0], y1 = v.y[k1], y2 = v.y[k2], y3 = v.y[k3];
    acc -= a0 * y0;
    acc -= a1 * y1;
    acc -= a2 * y2;
    acc -= a3 * y3;
  }
  for (; p < e; ++p) acc -= v.val[p] * v.y[ci[p]];
  v.y[i] = acc;
}
template <class T>
__device__ __forceinline__ void forward_row_warp(const EntryView<T> &v, int i, int lane) {
  const uint16_t *ci = v.ci();
  T part = T(0);
  for (int p = v.rp()[i] + lane, e = v.diag()[i]; p < e; p += 32) part += v.val[p] * v.y[ci[p]];
  part = butterfly_sum(part);
  if (lane == 0) v.y[i] -= part;
}

// Factors; with kY also y = L \ y.  Returns the first row with a bad pivot
// that this thread saw.  Ends with a barrier.  What a thread does in a level
// (its entry's words and first pair, or its row) does not depend on values:
// it is fetched in the level before.
template <class T, bool kY>
__device__ __forceinline__ unsigned factor_entries(const EntryView<T> &v) {
  const int tid = threadIdx.x, bd = blockDim.x, lane = tid & 31, nw = bd >> 5, rw = nw - 1 - (tid >> 5);
  T *const val = v.val, *const rd = v.rd;
  const int *eb = reinterpret_cast<const int *>(v.img + v.h.ebound);
  const int *fb = reinterpret_cast<const int *>(v.img + v.h.fbound);
  const uint2 *work = reinterpret_cast<const uint2 *>(v.img + v.h.work);
  const uint32_t *pair = v.img + v.h.pair;
  const uint16_t *frow = v.u16(v.h.frow);
  const int levels = v.h.levels;
  unsigned bad = 0xffffffffu;
  auto finish = [&](unsigned w, T acc) {
    const unsigned p = w & 0xffffu, aux = (w >> 16) & 0x3fffu, kind = w >> 30;
    if (kind == kEntryL) {
      val[p] = acc * rd[aux];
    } else if (kind != kEntryNone) {
      val[p] = acc;
      if (kind == kEntryPivot) {
        if (bad_value(acc)) bad = min(bad, aux);
        rd[aux] = pivot_reciprocal(acc);
      }
    }
  };
  // an entry's pairs from j on, four loads ahead of their multiply-adds
  auto pull = [&](T acc, unsigned j, unsigned e) {
    for (; j + 4 <= e; j += 4) {
      const uint32_t q0 = pair[j], q1 = pair[j + 1], q2 = pair[j + 2], q3 = pair[j + 3];
      const T l0 = val[q0 & 0xffffu], u0 = val[q0 >> 16], l1 = val[q1 & 0xffffu], u1 = val[q1 >> 16];
      const T l2 = val[q2 & 0xffffu], u2 = val[q2 >> 16], l3 = val[q3 & 0xffffu], u3 = val[q3 >> 16];
      acc -= l0 * u0;
      acc -= l1 * u1;
      acc -= l2 * u2;
      acc -= l3 * u3;
    }
    for (; j < e; ++j) {
      const uint32_t q = pair[j];
      acc -= val[q & 0xffffu] * val[q >> 16];
    }
    return acc;
  };
  int e0 = eb[0], e1 = eb[1], e2 = eb[2], f0 = 0, f1 = 0, f2 = 0;
  if (kY) {
    f0 = fb[0];
    f1 = fb[1];
    f2 = fb[2];
  }
  uint2 w{0, 0};
  uint32_t first = 0;
  int row = 0;
  auto fetch = [&]() {
    const int ns = e1 - e0;
    if (tid < ns) {
      w = work[e0 + tid];
      if (w.y >> 16) first = pair[w.y & 0xffffu];
    } else if (kY && tid < ns + f1 - f0) {
      row = frow[f0 + tid - ns];
    }
  };
  if (levels > 0) fetch();
  for (int lv = 0; lv < levels; ++lv) {
    const int ns = e1 - e0, c0 = e0, c1 = e1, c2 = e2, g0 = f0, g1 = f1, g2 = f2;
    if (tid < ns) {
      T acc = val[w.x & 0xffffu];
      const unsigned j = w.y & 0xffffu, c = w.y >> 16;
      if (c) {
        acc -= val[first & 0xffffu] * val[first >> 16];
        acc = pull(acc, j + 1, j + c);
      }
      finish(w.x, acc);
    } else if (kY && tid < ns + g1 - g0) {
      forward_row(v, row);
    }
    for (int k = tid + bd; k < ns + g1 - g0; k += bd) {
      if (k < ns) {
        const uint2 x = work[c0 + k];
        finish(x.x, pull(val[x.x & 0xffffu], x.y & 0xffffu, (x.y & 0xffffu) + (x.y >> 16)));
      } else if (kY) {
        forward_row(v, frow[g0 + k - ns]);
      }
    }
    for (int k = rw; k < c2 - c1 + g2 - g1; k += nw) {
      if (k < c2 - c1) {
        const uint2 x = work[c1 + k];
        T part = T(0);
        for (unsigned j = (x.y & 0xffffu) + lane, e = (x.y & 0xffffu) + (x.y >> 16); j < e; j += 32) {
          const uint32_t q = pair[j];
          part += val[q & 0xffffu] * val[q >> 16];
        }
        part = butterfly_sum(part);
        if (lane == 0) finish(x.x, val[x.x & 0xffffu] - part);
      } else if (kY) {
        forward_row_warp(v, frow[g1 + k - (c2 - c1)], lane);
      }
    }
    if (lv + 1 < levels) {
      e0 = c2;
      e1 = eb[2 * lv + 3];
      e2 = eb[2 * lv + 4];
      if (kY) {
        f0 = g2;
        f1 = fb[2 * lv + 3];
        f2 = fb[2 * lv + 4];
      }
      fetch();
    }
    __syncthreads();
  }
  return bad;
}

// y = L \ y alone, by the row levels.
template <class T>
__device__ __forceinline__ void forward_entries(const EntryView<T> &v) {
  const int tid = threadIdx.x, bd = blockDim.x, lane = tid & 31, nw = bd >> 5;
  const int *sb = reinterpret_cast<const int *>(v.img + v.h.sbound);
  const uint16_t *srow = v.u16(v.h.srow);
  for (int lv = 0; lv < v.h.slevels; ++lv) {
    const int s0 = sb[2 * lv], s1 = sb[2 * lv + 1], s2 = sb[2 * lv + 2];
    for (int k = s0 + tid; k < s1; k += bd) forward_row(v, srow[k]);
    for (int k = s1 + nw - 1 - (tid >> 5); k < s2; k += nw) forward_row_warp(v, srow[k], lane);
    __syncthreads();
  }
}

// y = U \ y in place: a row reads only rows of lower U levels.
template <class T>
__device__ __forceinline__ void backward_entries(const EntryView<T> &v) {
  const int tid = threadIdx.x, bd = blockDim.x, lane = tid & 31, nw = bd >> 5;
  const int *ub = reinterpret_cast<const int *>(v.img + v.h.ubound);
  const uint16_t *urow = v.u16(v.h.urow), *ci = v.ci(), *rp = v.rp(), *diag = v.diag();
  for (int lv = 0; lv < v.h.ulevels; ++lv) {
    const int s0 = ub[2 * lv], s1 = ub[2 * lv + 1], s2 = ub[2 * lv + 2];
    for (int k = s0 + tid; k < s1; k += bd) {
      const int i = urow[k];
      T acc = v.y[i];
      for (int p = diag[i] + 1, e = rp[i + 1]; p < e; ++p) acc -= v.val[p] * v.y[ci[p]];
      v.y[i] = acc * v.rd[i];
    }
    for (int k = s1 + nw - 1 - (tid >> 5); k < s2; k += nw) {
      const int i = urow[k];
      T part = T(0);
      for (int p = diag[i] + 1 + lane, e = rp[i + 1]; p < e; p += 32) part += v.val[p] * v.y[ci[p]];
      part = butterfly_sum(part);
      if (lane == 0) v.y[i] = (v.y[i] - part) * v.rd[i];
    }
    __syncthreads();
  }
}

}  // namespace xg
