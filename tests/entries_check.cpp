// Checks the entry schedule of a small factor (LuEntries, xg_lu.h) for the
// matrix in a file: positions within range, each entry and row placed once,
// nothing read before it is final, and the same factor and solution as a
// row-wise elimination.  Prints "ok <levels> <largest difference>".
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "xg_lu.h"

using namespace xg;

static void need(bool ok, const char *what) {
  if (!ok) {
    std::printf("FAIL: %s\n", what);
    std::exit(1);
  }
}

int main(int argc, char **argv) {
  need(argc > 2, "usage");
  FILE *f = std::fopen(argv[1], "rb");
  need(f, "open");
  int64_t head[2];
  need(std::fread(head, 8, 2, f) == 2, "read");
  const int n = int(head[0]);
  const int64_t nnz_a = head[1];
  std::vector<int> rp(n + 1), ci(nnz_a);
  std::vector<double> a(nnz_a);
  need(std::fread(rp.data(), 4, n + 1, f) == size_t(n + 1) && std::fread(ci.data(), 4, nnz_a, f) == size_t(nnz_a) &&
           std::fread(a.data(), 8, nnz_a, f) == size_t(nnz_a), "read");
  std::fclose(f);
  LuSymbolic S;
  std::string err;
  need(!lu_analyze(n, rp.data(), ci.data(), a.data(), 1e-3, &S, &err, std::atoi(argv[2])), err.c_str());
  need(lu_build_updates(S), "updates");
  LuEntries E;
  if (!lu_build_entries(S, &E)) {
    std::printf("no schedule\n");
    return 0;
  }
  const LuEntriesHead &h = E.head;
  const uint32_t *img = E.image.data();
  auto u16 = [&](int w) { return reinterpret_cast<const uint16_t *>(img + w); };
  auto bound = [&](int w, int k) { return int(img[w + k]); };
  need(h.words == int(E.image.size()) && h.factor <= h.both && h.solve0 <= h.both && h.both <= h.words, "parts");
  for (int w : {h.factor, h.solve0, h.both, h.words, h.work, h.pair}) need(w % 4 == 0, "16-byte parts");
  need(h.work < h.factor && h.pair <= h.factor && h.ebound < h.factor && h.ci >= h.solve0 && h.rp >= h.solve0 &&
           h.diag >= h.solve0 && h.ubound < h.both && h.urow < h.both && h.fbound < h.both && h.frow < h.both &&
           h.urow >= h.solve0, "what each mode stages");
  const int nnz = S.rp[n];
  for (int p = 0; p < nnz; ++p) need(u16(h.ci)[p] == S.ci[p], "columns");
  for (int i = 0; i < n; ++i) need(u16(h.rp)[i] == S.rp[i] && u16(h.diag)[i] == S.diag[i], "rows");
  need(u16(h.rp)[n] == nnz, "row end");
  std::vector<double> v(nnz), w(nnz), rd(n, 0.0), y(n), z(n);
  std::vector<int> done(nnz, 0), rdone(n, 0), ydone(n, 0);
  for (int p = 0; p < nnz; ++p) v[p] = w[p] = S.lu2a[p] >= 0 ? a[S.lu2a[p]] : 0.0;
  for (int i = 0; i < n; ++i) y[i] = z[i] = std::cos(1.0 + i);
  // entries with no work and rows with no L part are final from the start
  std::vector<char> has(nnz, 0);
  for (int t = 0; t < h.n_work; ++t)
    if (img[h.work + 2 * t] >> 30 != kEntryNone) has[img[h.work + 2 * t] & 0xffffu] += 1;
  for (int p = 0; p < nnz; ++p) {
    need(has[p] <= 1, "entry once");
    done[p] = !has[p];
  }
  for (int i = 0; i < n; ++i) ydone[i] = S.diag[i] == S.rp[i];
  int most = 0;
  for (int lv = 0; lv < h.levels; ++lv) {
    std::vector<int> newp, newr, newy;
    const int e0 = bound(h.ebound, 2 * lv), e1 = bound(h.ebound, 2 * lv + 1), e2 = bound(h.ebound, 2 * lv + 2);
    need(e0 <= e1 && e1 <= e2 && e2 <= h.n_work, "entry bounds");
    most = std::max(most, e2 - e0);
    for (int t = e0; t < e2; ++t) {
      const uint32_t w0 = img[h.work + 2 * t], w1 = img[h.work + 2 * t + 1];
      const int p = w0 & 0xffffu, aux = (w0 >> 16) & 0x3fffu, kind = w0 >> 30, j0 = w1 & 0xffffu, c = w1 >> 16;
      need(p < nnz && j0 + c <= h.n_pair && (c > kEntryLong) == (t >= e1), "entry");
      if (t > e0 && (t - e0) % 32 && t < e1)
        need(kind == int(img[h.work + 2 * t - 2] >> 30) || kind == int(kEntryNone), "a kind starts a warp");
      if (kind == int(kEntryNone)) {
        need(c == 0, "an idle place");
        continue;
      }
      double acc = v[p];
      for (int j = j0; j < j0 + c; ++j) {
        const int l = img[h.pair + j] & 0xffffu, u = img[h.pair + j] >> 16;
        need(l < nnz && u < nnz && done[l] && done[u], "pair read before it is final");
        acc -= v[l] * v[u];
      }
      if (kind == int(kEntryL)) {
        need(aux < n && rdone[aux], "pivot read before it is final");
        v[p] = acc * rd[aux];
      } else {
        v[p] = acc;
        if (kind == int(kEntryPivot)) {
          need(aux < n && S.diag[aux] == p, "pivot row");
          rd[aux] = 1 / acc;
          newr.push_back(aux);
        }
      }
      newp.push_back(p);
    }
    for (int k = bound(h.fbound, 2 * lv); k < bound(h.fbound, 2 * lv + 2); ++k) {
      const int i = u16(h.frow)[k];
      need(i < n && !ydone[i] && (S.diag[i] - S.rp[i] > kEntryLong) == (k >= bound(h.fbound, 2 * lv + 1)), "row");
      for (int p = S.rp[i]; p < S.diag[i]; ++p) {
        need(done[p] && ydone[S.ci[p]], "row before its inputs");
        y[i] -= v[p] * y[S.ci[p]];
      }
      newy.push_back(i);
    }
    for (int p : newp) done[p] = 1;
    for (int i : newr) rdone[i] = 1;
    for (int i : newy) ydone[i] = 1;
  }
  for (int p = 0; p < nnz; ++p) need(done[p], "every entry");
  for (int i = 0; i < n; ++i) need(rdone[i] && ydone[i], "every row");
  need(h.max_width == most, "widest level");
  // forward by row levels
  std::vector<double> y2(n);
  std::vector<int> sdone(n, 0);
  for (int i = 0; i < n; ++i) {
    y2[i] = std::cos(1.0 + i);
    sdone[i] = S.diag[i] == S.rp[i];
  }
  for (int lv = 0; lv < h.slevels; ++lv) {
    std::vector<int> now;
    for (int k = bound(h.sbound, 2 * lv); k < bound(h.sbound, 2 * lv + 2); ++k) {
      const int i = u16(h.srow)[k];
      for (int p = S.rp[i]; p < S.diag[i]; ++p) {
        need(sdone[S.ci[p]], "solve row before its inputs");
        y2[i] -= v[p] * y2[S.ci[p]];
      }
      now.push_back(i);
    }
    for (int i : now) sdone[i] = 1;
  }
  need(y == y2, "forward solves agree");
  // backward
  std::vector<int> udone(n, 0);
  for (int lv = 0; lv < h.ulevels; ++lv) {
    std::vector<int> now;
    for (int k = bound(h.ubound, 2 * lv); k < bound(h.ubound, 2 * lv + 2); ++k) {
      const int i = u16(h.urow)[k];
      for (int p = S.diag[i] + 1; p < S.rp[i + 1]; ++p) {
        need(udone[S.ci[p]], "backward row before its inputs");
        y[i] -= v[p] * y[S.ci[p]];
      }
      y[i] *= rd[i];
      now.push_back(i);
    }
    for (int i : now) udone[i] = 1;
  }
  // row-wise elimination
  std::vector<double> rw(n);
  for (int i = 0; i < n; ++i) {
    int64_t u = S.urp[i];
    for (int p = S.rp[i]; p < S.diag[i]; ++p) {
      const int k = S.ci[p];
      w[p] *= rw[k];
      for (int q = S.diag[k] + 1; q < S.rp[k + 1]; ++q) w[S.upos[size_t(u++)]] -= w[p] * w[q];
    }
    rw[i] = 1 / w[S.diag[i]];
  }
  double diff = 0;
  for (int p = 0; p < nnz; ++p) diff = std::max(diff, std::fabs(v[p] - w[p]));
  for (int i = 0; i < n; ++i) {
    need(udone[i], "every backward row");
    for (int p = S.rp[i]; p < S.diag[i]; ++p) z[i] -= w[p] * z[S.ci[p]];
  }
  for (int i = n - 1; i >= 0; --i) {
    for (int p = S.diag[i] + 1; p < S.rp[i + 1]; ++p) z[i] -= w[p] * z[S.ci[p]];
    z[i] *= rw[i];
    diff = std::max(diff, std::fabs(z[i] - y[i]));
  }
  std::printf("ok %d %.3g entries %d work %d pairs %d widest %d row levels %d %d words %d\n", h.levels, diff, nnz, h.n_work,
              h.n_pair, h.max_width, h.slevels, h.ulevels, h.words);
  return 0;
}
