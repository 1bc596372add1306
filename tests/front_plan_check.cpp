// Checks the multifrontal plan (lu_front.h) of the matrix in a file: every
// index the kernels follow lies in its buffer, every entry of A lands once,
// and the elimination and solves over the plan's maps, done here as the
// kernels do them, solve the system.  Prints "ok <backward error>".
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "lu_front.h"

using namespace xg;

static void need(bool ok, const char *what) {
  if (!ok) {
    std::printf("FAIL: %s\n", what);
    std::exit(1);
  }
}

int main(int argc, char **argv) {
  need(argc > 1, "usage");
  FILE *f = std::fopen(argv[1], "rb");
  need(f, "open");
  int64_t head[2];
  need(std::fread(head, 8, 2, f) == 2, "read");
  const int n = int(head[0]);
  const int64_t nnz = head[1];
  std::vector<int> rp(n + 1), ci(nnz);
  std::vector<double> a(nnz);
  need(std::fread(rp.data(), 4, n + 1, f) == size_t(n + 1) && std::fread(ci.data(), 4, nnz, f) == size_t(nnz) &&
           std::fread(a.data(), 8, nnz, f) == size_t(nnz), "read");
  std::fclose(f);
  LuSymbolic S;
  std::string err;
  need(!lu_analyze(n, rp.data(), ci.data(), a.data(), 1e-3, &S, &err, 0), err.c_str());
  FrontPlan P;
  if (!build_front_plan(S, rp.data(), ci.data(), &P)) {
    std::printf("no plan\n");
    return 0;
  }
  const int nf = int(P.front.size());
  need(P.inv.size() == P.child.size(), "inverse maps");
  // every unknown has one place: in a front's pivots or in the rows outside
  std::vector<int> seen(n, 0), used(nnz, 0);
  for (auto *R : {&P.before, &P.after})
    for (size_t i = 0; i < R->row.size(); ++i) {
      ++seen[R->row[i]];
      need(R->diag[i] >= 0, "pivot entry");
      ++used[R->diag[i]];
    }
  for (auto *R : {&P.before, &P.core, &P.after}) {
    if (R->ptr.empty()) continue;
    need(R->ptr.size() == R->row.size() + 1 && R->ptr.back() == int64_t(R->col.size()), "row starts");
    need(R->round.back() == int(R->row.size()), "rounds");
    for (size_t k = 0; k + 2 < R->round.size(); k += 2)
      for (int i = R->round[k]; i < R->round[k + 2]; ++i)
        need((R->ptr[i + 1] - R->ptr[i] > kFrontLongRow) == (i < R->round[k + 1]), "long rows first");
    for (size_t e = 0; e < R->col.size(); ++e) {
      need(R->col[e] >= 0 && R->col[e] < n, "row column");
      ++used[R->a[e]];
    }
  }
  int64_t nl = 0, nu = 0, nc = 0, np = 0, nb = 0;
  for (int s = 0; s < nf; ++s) {
    const Front &F = P.front[s];
    const int64_t b = F.m - F.p;
    need(F.p > 0 && F.m >= F.p && F.m <= kFrontMax, "front size");
    need(F.lo == nl && F.uo == nu && F.co == nc && F.pv == np && F.bv == nb, "front places");
    nl += int64_t(F.m) * F.p; nu += b * F.p; nc += b * b; np += F.p; nb += b;
    need(F.idx + F.m <= int64_t(P.idx.size()), "front unknowns");
    for (int k = 0; k < F.m; ++k) need(P.idx[F.idx + k] >= 0 && P.idx[F.idx + k] < n, "unknown");
    for (int k = 0; k < F.p; ++k) ++seen[P.idx[F.idx + k]];
    need(F.child1 - F.child0 <= kFrontMaxChildren, "children");
    for (int c = F.child0; c < F.child1; ++c) {
      const Front &G = P.front[P.child[c]];
      need(G.level < F.level && P.child[c] < s && G.parent == s, "child before parent");
      need(P.inv[c] + F.m <= int64_t(P.inv_map.size()) && G.map + G.m - G.p <= int64_t(P.map.size()), "map places");
      for (int k = 0; k < G.m - G.p; ++k) {
        const int at = P.map[G.map + k];
        need(at >= 0 && at < F.m && P.inv_map[P.inv[c] + at] == k, "maps are inverse");
        need(P.idx[F.idx + at] == P.idx[G.idx + G.p + k], "map keeps the unknown");
      }
      int back = 0;
      for (int k = 0; k < F.m; ++k) back += P.inv_map[P.inv[c] + k] >= 0;
      need(back == G.m - G.p, "inverse map size");
    }
    need(F.acol + F.na <= int64_t(P.apos.size()) && P.apos.size() == P.aidx.size(), "A entries");
    for (int64_t e = F.acol; e < F.acol + F.na; ++e) {
      const int i = P.apos[e] % kFrontMax, j = P.apos[e] / kFrontMax;
      need(i < F.m && j < F.m && (j < F.p || i < F.p), "A entry place");
      ++used[P.aidx[e]];
    }
  }
  need(nl == P.n_l && nu == P.n_u && nc == P.n_c && np == P.n_pv && nb == P.n_bv, "buffer sizes");
  for (int k = 0; k < n; ++k) need(seen[k] == 1, "each unknown once");
  for (int64_t e = 0; e < nnz; ++e) need(used[e] == 1, "each A entry once");
  for (size_t l = 0; l + 1 < P.level.size(); ++l)
    for (int s = P.level[l]; s < P.level[l + 1]; ++s) {
      need(P.front[s].level == int(l), "levels");
      auto size_class = [](int m) { return m > kFrontMiddle ? 0 : m > kFrontLow ? 1 : 2; };
      need(s == P.level[l] || size_class(P.front[s].m) >= size_class(P.front[s - 1].m), "size classes in order");
    }

  // eliminate
  std::vector<double> L(P.n_l), U(P.n_u), C(P.n_c), rd(P.n_pv), y(P.n_pv), bv(P.n_bv), xk(n, 0.0), x(n, 0.0), rhs(n);
  double most = 0;
  for (int s = 0; s < nf; ++s) {
    const Front &F = P.front[s];
    const int m = F.m, p = F.p, b = m - p;
    std::vector<double> W(size_t(m) * m, 0.0);
    for (int64_t e = F.acol; e < F.acol + F.na; ++e)
      W[P.apos[e] % kFrontMax + size_t(P.apos[e] / kFrontMax) * m] = a[P.aidx[e]];
    for (int c = F.child0; c < F.child1; ++c) {
      const Front &G = P.front[P.child[c]];
      const int g = G.m - G.p;
      for (int j = 0; j < m; ++j) {
        const int jc = P.inv_map[P.inv[c] + j];
        if (jc < 0) continue;
        for (int i = 0; i < g; ++i) W[P.map[G.map + i] + size_t(j) * m] += C[G.co + i + int64_t(jc) * g];
      }
    }
    for (int k = 0; k < p; ++k) {
      need(W[k + size_t(k) * m] != 0.0, "pivot");
      rd[F.pv + k] = 1 / W[k + size_t(k) * m];
      for (int i = k + 1; i < m; ++i) {
        W[i + size_t(k) * m] *= rd[F.pv + k];
        most = std::max(most, std::fabs(W[i + size_t(k) * m]));
      }
      for (int j = k + 1; j < m; ++j)
        for (int i = k + 1; i < m; ++i) W[i + size_t(j) * m] -= W[i + size_t(k) * m] * W[k + size_t(j) * m];
    }
    for (int j = 0; j < p; ++j)
      for (int i = 0; i < m; ++i) L[F.lo + i + int64_t(j) * m] = W[i + size_t(j) * m];
    for (int j = 0; j < b; ++j) {
      for (int i = 0; i < p; ++i) U[F.uo + i + int64_t(j) * p] = W[i + size_t(p + j) * m];
      for (int i = 0; i < b; ++i) C[F.co + i + int64_t(j) * b] = W[p + i + size_t(p + j) * m];
    }
  }
  // solve
  for (int i = 0; i < n; ++i) rhs[i] = std::sin(1.0 + i);
  auto rows = [&](const FrontRows &R) {
    for (size_t i = 0; i < R.row.size(); ++i) {
      double v = rhs[S.P[R.row[i]]];
      for (int64_t e = R.ptr[i]; e < R.ptr[i + 1]; ++e) v -= a[R.a[e]] * xk[R.col[e]];
      if (R.diag[i] >= 0) x[P.Q[R.row[i]]] = v /= a[R.diag[i]];
      xk[R.row[i]] = v;
    }
  };
  rows(P.before);
  rows(P.core);
  for (int s = 0; s < nf; ++s) {
    const Front &F = P.front[s];
    std::vector<double> v(F.m, 0.0);
    for (int i = 0; i < F.m; ++i) {
      for (int c = F.child0; c < F.child1; ++c) {
        const int at = P.inv_map[P.inv[c] + i];
        if (at >= 0) v[i] += bv[P.front[P.child[c]].bv + at];
      }
      if (i < F.p) v[i] += xk[P.idx[F.idx + i]];
    }
    for (int k = 0; k < F.p; ++k)
      for (int i = k + 1; i < F.m; ++i) v[i] -= L[F.lo + i + int64_t(k) * F.m] * v[k];
    for (int k = 0; k < F.p; ++k) y[F.pv + k] = v[k];
    for (int k = F.p; k < F.m; ++k) bv[F.bv + k - F.p] = v[k];
  }
  for (int s = nf - 1; s >= 0; --s) {
    const Front &F = P.front[s];
    std::vector<double> v(F.p);
    for (int i = 0; i < F.p; ++i) {
      v[i] = y[F.pv + i];
      for (int j = 0; j < F.m - F.p; ++j) v[i] -= U[F.uo + i + int64_t(j) * F.p] * xk[P.idx[F.idx + F.p + j]];
    }
    for (int k = F.p - 1; k >= 0; --k) {
      v[k] *= rd[F.pv + k];
      for (int i = 0; i < k; ++i) v[i] -= L[F.lo + i + int64_t(k) * F.m] * v[k];
      const int u = P.idx[F.idx + k];
      xk[u] = x[P.Q[u]] = v[k];
    }
  }
  rows(P.after);
  double r = 0, an = 0, xn = 0;
  for (int i = 0; i < n; ++i) {
    double t = rhs[i], w = 0;
    for (int p = rp[i]; p < rp[i + 1]; ++p) {
      t -= a[p] * x[ci[p]];
      w += std::fabs(a[p]);
    }
    r = std::max(r, std::fabs(t));
    an = std::max(an, w);
    xn = std::max(xn, std::fabs(x[i]));
  }
  std::printf("ok %.3g fronts %d levels %zu flops %.3g multiplier %.3g before %zu after %zu\n", r / (an * xn + 1.0), nf,
              P.level.size() - 1, P.flops, most, P.before.row.size(), P.after.row.size());
  return 0;
}
