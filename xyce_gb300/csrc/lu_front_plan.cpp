// lu_front_plan.cpp — builds the multifrontal plan (lu_front.h): singletons, a
// nested-dissection order with refined separators, the symbolic elimination
// on the pattern of B + B^T, fronts and their index maps.

#include "lu_front.h"

#include <algorithm>
#include <cmath>
#include <numeric>

namespace xg {
namespace {

struct Graph {
  std::vector<int> ptr, adj;
};

constexpr int kLeaf = 60;            // parts of at most this many vertices: minimum degree
constexpr double kMinShare = 0.3;    // a separator leaves each side at least this share
constexpr double kMaxShare = 0.62;   // and its refinement at most this one
constexpr int kRefinePasses = 6;
constexpr int kRefineSteps = 1000;
constexpr int kRefineLimit = 4000;   // separators larger than this are taken as they come

// Nested dissection by level structures (George and Liu, 1981) whose
// separator is then refined by moving its vertices to either side (the
// vertex form of Fiduccia and Mattheyses, "A linear-time heuristic for
// improving network partitions", DAC 1982: best gain first, each vertex
// once, the best prefix of the moves kept).  On a 200,000-transistor block
// of random logic the refinement halves the separators: 445M to 189M
// multiply-adds.
class Dissection {
 public:
  explicit Dissection(const Graph &g)
      : g_(g), n_(int(g.ptr.size()) - 1), in_(n_, 0), level_(n_, -1), local_(n_, -1), side_(n_, 0) {}

  std::vector<int> order() {
    const int dense = std::max(16, int(10.0 * std::sqrt(double(n_))));
    std::vector<int> all, last;
    for (int i = 0; i < n_; ++i) (g_.ptr[i + 1] - g_.ptr[i] > dense ? last : all).push_back(i);
    work_.push_back({false, std::move(all)});
    while (!work_.empty()) {
      Part part = std::move(work_.back());
      work_.pop_back();
      if (part.emit) out_.insert(out_.end(), part.v.begin(), part.v.end());
      else if (int(part.v.size()) <= kLeaf) leaf(part.v);
      else split(part.v);
    }
    out_.insert(out_.end(), last.begin(), last.end());
    return std::move(out_);
  }

 private:
  struct Part {
    bool emit;
    std::vector<int> v;
  };
  enum Side : char { A = 1, B = 2, SEP = 3 };

  void leaf(const std::vector<int> &v) {
    const int m = int(v.size());
    for (int k = 0; k < m; ++k) local_[v[k]] = k;
    std::vector<int> p(m + 1, 0), j;
    for (int k = 0; k < m; ++k) {
      for (int e = g_.ptr[v[k]]; e < g_.ptr[v[k] + 1]; ++e)
        if (local_[g_.adj[e]] >= 0) j.push_back(local_[g_.adj[e]]);
      p[k + 1] = int(j.size());
    }
    for (int k : amd_order(m, p.data(), j.data(), nullptr)) out_.push_back(v[k]);
    for (int u : v) local_[u] = -1;
  }

  // Breadth-first levels of the members (in_ == stamp) from root, in q.
  void levels(int root, int stamp, std::vector<int> &q) {
    q.assign(1, root);
    level_[root] = 0;
    in_[root] = -stamp;
    for (size_t h = 0; h < q.size(); ++h) {
      const int u = q[h];
      for (int e = g_.ptr[u]; e < g_.ptr[u + 1]; ++e) {
        const int v = g_.adj[e];
        if (in_[v] != stamp) continue;
        in_[v] = -stamp;
        level_[v] = level_[u] + 1;
        q.push_back(v);
      }
    }
  }

  void split(const std::vector<int> &V) {
    const int stamp = ++stamp_;
    for (int u : V) in_[u] = stamp;
    std::vector<int> q;
    int root = V[0], ecc = -1;
    for (int tries = 0; tries < 6; ++tries) {
      levels(root, stamp, q);
      for (int u : q) in_[u] = stamp;
      const int e = level_[q.back()];
      if (e <= ecc) break;
      ecc = e;
      int best = q.back(), bd = n_ + 1;
      for (int k = int(q.size()) - 1; k >= 0 && level_[q[k]] == e; --k) {
        const int d = g_.ptr[q[k] + 1] - g_.ptr[q[k]];
        if (d < bd) {
          bd = d;
          best = q[k];
        }
      }
      root = best;
    }
    levels(root, stamp, q);
    if (q.size() < V.size()) {
      // several components: each is a part of its own, the small ones together
      std::vector<int> small;
      auto part = [&](std::vector<int> c) {
        if (int(c.size()) <= kLeaf) small.insert(small.end(), c.begin(), c.end());
        else work_.push_back({false, std::move(c)});
      };
      part(q);
      for (int u : V)
        if (in_[u] == stamp) {
          levels(u, stamp, q);
          part(q);
        }
      for (int u : V) level_[u] = -1;
      if (!small.empty()) leaf(small);
      return;
    }
    for (int u : V) in_[u] = stamp;
    const int h = level_[q.back()] + 1, N = int(V.size());
    // the level whose vertices with a neighbour in the next one are fewest,
    // among those that leave both sides their share
    std::vector<int> count(h, 0), cut(h, 0);
    auto cuts = [&](int u) {
      for (int e = g_.ptr[u]; e < g_.ptr[u + 1]; ++e)
        if (in_[g_.adj[e]] == stamp && level_[g_.adj[e]] == level_[u] + 1) return true;
      return false;
    };
    for (int u : V) {
      ++count[level_[u]];
      if (cuts(u)) ++cut[level_[u]];
    }
    int at = -1;
    double best = 0;
    for (int c = 1, below = count[0]; c < h - 1; ++c) {
      below += count[c];
      const int a = below - cut[c], b = N - below;
      if (a <= 0 || b <= 0) continue;
      const double share = double(std::min(a, b)) / N;
      const double cost = cut[c] * (1 + 0.4 * (0.5 - share)) + (share >= kMinShare ? 0.0 : 1e6 * (kMinShare - share));
      if (at < 0 || cost < best) {
        best = cost;
        at = c;
      }
    }
    if (at < 0) {  // too shallow to split: a near-clique
      for (int u : V) level_[u] = -1;
      leaf(V);
      return;
    }
    int na = 0, nb = 0, ns = 0;
    for (int u : V) {
      side_[u] = level_[u] > at ? B : level_[u] == at && cuts(u) ? SEP : A;
      ++(side_[u] == A ? na : side_[u] == B ? nb : ns);
    }
    for (int pass = 0; pass < kRefinePasses && ns <= kRefineLimit; ++pass)
      if (!refine(V, stamp, N, na, nb, ns)) break;
    std::vector<int> va, vb, vs;
    for (int u : V) {
      (side_[u] == A ? va : side_[u] == B ? vb : vs).push_back(u);
      level_[u] = -1;
    }
    if (va.empty() || vb.empty()) {
      leaf(V);
      return;
    }
    work_.push_back({true, std::move(vs)});
    work_.push_back({false, std::move(vb)});
    work_.push_back({false, std::move(va)});
  }

  // One pass of separator moves; false when it found nothing better.
  bool refine(const std::vector<int> &V, int stamp, int N, int &na, int &nb, int &ns) {
    constexpr int kMoved = -7;  // local_ of a vertex that has moved in this pass
    std::vector<int> sep, moved;
    for (int u : V)
      if (side_[u] == SEP) sep.push_back(u);
    std::vector<std::pair<int, char>> log;  // vertex, the side it came from
    auto count_of = [&](char s) -> int & { return s == A ? na : s == B ? nb : ns; };
    int best_ns = ns, best_gap = std::abs(na - nb), idle = 0;
    size_t keep = 0;
    for (int step = 0; step < kRefineSteps && idle < 50; ++step) {
      int bu = -1, bg = -4, bbal = 0;
      char bto = A;
      for (size_t x = 0; x < sep.size();) {
        const int u = sep[x];
        if (side_[u] != SEP || local_[u] == kMoved) {
          sep[x] = sep.back();
          sep.pop_back();
          continue;
        }
        int to_a = 1, to_b = 1;  // what the separator loses when u goes to A / to B
        for (int e = g_.ptr[u]; e < g_.ptr[u + 1]; ++e) {
          const int v = g_.adj[e];
          if (in_[v] != stamp) continue;
          if (side_[v] == B) --to_a;
          else if (side_[v] == A) --to_b;
        }
        for (char to : {A, B}) {
          const int mine = count_of(to), other = count_of(to == A ? B : A);
          if (mine + 1 > kMaxShare * N && mine + 1 >= other) continue;
          const int gain = to == A ? to_a : to_b;
          if (gain > bg || (gain == bg && bu >= 0 && other - mine > bbal)) {
            bg = gain;
            bu = u;
            bto = to;
            bbal = other - mine;
          }
        }
        ++x;
      }
      if (bu < 0) break;
      log.push_back({bu, SEP});
      side_[bu] = bto;
      local_[bu] = kMoved;
      moved.push_back(bu);
      --ns;
      ++count_of(bto);
      const char away = bto == A ? B : A;
      for (int e = g_.ptr[bu]; e < g_.ptr[bu + 1]; ++e) {
        const int v = g_.adj[e];
        if (in_[v] != stamp || side_[v] != away) continue;
        log.push_back({v, away});
        side_[v] = SEP;
        ++ns;
        --count_of(away);
        sep.push_back(v);
      }
      if (ns < best_ns || (ns == best_ns && std::abs(na - nb) < best_gap)) {
        best_ns = ns;
        best_gap = std::abs(na - nb);
        keep = log.size();
        idle = 0;
      } else {
        ++idle;
      }
    }
    for (size_t x = log.size(); x-- > keep;) {
      --count_of(side_[log[x].first]);
      side_[log[x].first] = log[x].second;
      ++count_of(log[x].second);
    }
    for (int u : moved) local_[u] = -1;
    return keep > 0;
  }

  const Graph &g_;
  int n_, stamp_ = 0;
  std::vector<int> in_, level_, local_, out_;
  std::vector<char> side_;
  std::vector<Part> work_;
};

// B = A(P, Q) by rows and by columns, each entry with its place in A.
struct Matched {
  std::vector<int64_t> rp, cp;
  std::vector<int> rcol, ra, crow, ca;
};

Matched match(int n, const std::vector<int> &P, const std::vector<int> &Q, const int *rp, const int *ci) {
  std::vector<int> qinv(n);
  for (int k = 0; k < n; ++k) qinv[Q[k]] = k;
  Matched B;
  B.rp.assign(n + 1, 0);
  B.cp.assign(n + 1, 0);
  for (int k = 0; k < n; ++k) {
    B.rp[k + 1] = B.rp[k] + rp[P[k] + 1] - rp[P[k]];
    for (int p = rp[P[k]]; p < rp[P[k] + 1]; ++p) ++B.cp[qinv[ci[p]] + 1];
  }
  for (int k = 0; k < n; ++k) B.cp[k + 1] += B.cp[k];
  B.rcol.resize(B.rp[n]);
  B.ra.resize(B.rp[n]);
  B.crow.resize(B.rp[n]);
  B.ca.resize(B.rp[n]);
  std::vector<int64_t> fill(B.cp.begin(), B.cp.end() - 1);
  for (int k = 0; k < n; ++k) {
    int64_t q = B.rp[k];
    for (int p = rp[P[k]]; p < rp[P[k] + 1]; ++p, ++q) {
      const int c = qinv[ci[p]];
      B.rcol[q] = c;
      B.ra[q] = p;
      B.crow[fill[c]] = k;
      B.ca[fill[c]++] = p;
    }
  }
  return B;
}

enum Kind : char { CORE = 0, BEFORE = 1, AFTER = 2 };
constexpr int kRounds = 4;  // of singletons: a long chain of them is better left to the tree

// Pairs the rows of A with columns: singletons with their one entry (rows
// and columns come out in rounds, by row of A), the others with their
// diagonal entry where there is one.  False when A is structurally singular.
bool pair_rows(int n, const int *rp, const int *ci, std::vector<int> *col_of, std::vector<char> *kind_of,
               std::vector<std::vector<int>> *first, std::vector<std::vector<int>> *last) {
  std::vector<int> cp(n + 1, 0), cr(size_t(rp[n]));
  for (int p = 0; p < rp[n]; ++p) ++cp[ci[p] + 1];
  for (int c = 0; c < n; ++c) cp[c + 1] += cp[c];
  {
    std::vector<int> fill(cp.begin(), cp.end() - 1);
    for (int r = 0; r < n; ++r)
      for (int p = rp[r]; p < rp[r + 1]; ++p) cr[fill[ci[p]]++] = r;
  }
  std::vector<int> &col = *col_of, row_of(n, -1), rows_left(n), cols_left(n);
  std::vector<char> &kind = *kind_of;
  col.assign(n, -1);
  kind.assign(n, CORE);
  for (int k = 0; k < n; ++k) {
    rows_left[k] = rp[k + 1] - rp[k];
    cols_left[k] = cp[k + 1] - cp[k];
  }
  auto take = [&](int r, int c, char as) {
    kind[r] = as;
    col[r] = c;
    row_of[c] = r;
    for (int p = rp[r]; p < rp[r + 1]; ++p) --cols_left[ci[p]];
    for (int p = cp[c]; p < cp[c + 1]; ++p) --rows_left[cr[p]];
  };
  // the one entry left of a row (its column not taken) or of a column
  auto open_col = [&](int r) {
    for (int p = rp[r]; p < rp[r + 1]; ++p)
      if (row_of[ci[p]] < 0) return ci[p];
    return -1;
  };
  auto open_row = [&](int c) {
    for (int p = cp[c]; p < cp[c + 1]; ++p)
      if (col[cr[p]] < 0) return cr[p];
    return -1;
  };
  for (int round = 0; round < kRounds; ++round) {
    std::vector<std::pair<int, int>> r, c;
    std::vector<char> claimed(n, 0);
    for (int k = 0; k < n; ++k)
      if (col[k] < 0 && rows_left[k] == 1) {
        const int j = open_col(k);
        if (j >= 0 && !claimed[j]) {  // two rows with the same one column: singular, left to the tree
          claimed[j] = 1;
          r.push_back({k, j});
        }
      }
    for (auto &e : r) take(e.first, e.second, BEFORE);
    std::fill(claimed.begin(), claimed.end(), 0);
    for (int k = 0; k < n; ++k)
      if (row_of[k] < 0 && cols_left[k] == 1) {
        const int j = open_row(k);
        if (j >= 0 && !claimed[j]) {
          claimed[j] = 1;
          c.push_back({j, k});
        }
      }
    for (auto &e : c) take(e.first, e.second, AFTER);
    if (r.empty() && c.empty()) break;
    std::vector<int> rows;
    for (auto &e : r) rows.push_back(e.first);
    if (!rows.empty()) first->push_back(rows);
    rows.clear();
    for (auto &e : c) rows.push_back(e.first);
    if (!rows.empty()) last->push_back(rows);
  }
  // the rest: the diagonal where it is an entry, then an augmenting path for
  // each row that lacks it (a maximum transversal, Duff, "On algorithms for
  // obtaining a maximum transversal", ACM TOMS 7(3), 1981)
  std::vector<int> open;
  for (int r = 0; r < n; ++r) {
    if (col[r] >= 0) continue;
    if (row_of[r] < 0 && std::binary_search(ci + rp[r], ci + rp[r + 1], r)) {
      col[r] = r;
      row_of[r] = r;
    } else {
      open.push_back(r);
    }
  }
  std::vector<int> seen(n, -1), at(n, 0), path;
  for (int r : open) {
    path.assign(1, r);
    at[r] = rp[r];
    bool done = false;
    while (!path.empty() && !done) {
      const int u = path.back();
      int next = -1;
      for (int p = rp[u]; p < rp[u + 1] && !done; ++p)  // a free column ends the path
        if (row_of[ci[p]] < 0) {
          at[u] = p;
          done = true;
        }
      if (done) break;
      while (at[u] < rp[u + 1] && next < 0) {
        const int c = ci[at[u]];
        if (seen[c] != r && kind[row_of[c]] == CORE) {
          seen[c] = r;
          next = row_of[c];
        } else {
          ++at[u];
        }
      }
      if (next < 0) {
        path.pop_back();
        if (!path.empty()) ++at[path.back()];
        continue;
      }
      path.push_back(next);
      at[next] = rp[next];
    }
    if (!done) return false;
    for (int u : path) {
      col[u] = ci[at[u]];
      row_of[col[u]] = u;
    }
  }
  return true;
}

// Adds rows (one round) with the entries pick(column) accepts.
template <class F>
void add_round(FrontRows &R, const Matched &B, std::vector<int> rows, bool solved, F pick) {
  if (R.ptr.empty()) R.ptr.push_back(0);
  if (R.round.empty()) R.round.push_back(0);
  auto length = [&](int k) {
    int64_t c = 0;
    for (int64_t q = B.rp[k]; q < B.rp[k + 1]; ++q) c += B.rcol[q] != k && pick(B.rcol[q]);
    return c;
  };
  auto mid = std::stable_partition(rows.begin(), rows.end(), [&](int k) { return length(k) > kFrontLongRow; });
  const int n_long = int(mid - rows.begin());
  for (int k : rows) {
    int diag = -1;
    for (int64_t q = B.rp[k]; q < B.rp[k + 1]; ++q) {
      const int c = B.rcol[q];
      if (c == k) {
        diag = B.ra[q];
      } else if (pick(c)) {
        R.col.push_back(c);
        R.a.push_back(B.ra[q]);
      }
    }
    R.row.push_back(k);
    R.diag.push_back(solved ? diag : -1);
    R.ptr.push_back(int64_t(R.col.size()));
  }
  R.round.push_back(R.round.back() + n_long);
  R.round.push_back(int(R.row.size()));
}

// A front being built: pivots and border are positions in the elimination order.
struct Draft {
  std::vector<int> piv, border, child;
  double work0 = 0;  // multiply-adds of the columns it was made of
  int parent = -1, level = 0;
  bool gone = false;
};

constexpr double kModelSms = 152.0;  // SMs of the GB300 whose times the model below follows
constexpr int kSmallPivots = 16, kSmallRows = 48;
constexpr double kSmallGrowth = 4.0, kGrowth = 0.2;

// Merges children into their parents where that adds little work: at most
// 20% over the columns' own, or up to 5x for fronts of at most 16 pivots and
// 48 rows (one warp's or two's work either way).
void merge_fronts(std::vector<Draft> &F, const std::vector<int> &by_pivot) {
  for (int i : by_pivot) {
    for (;;) {
      int best = -1;
      double best_growth = 0;
      for (int c : F[i].child) {
        const double p = double(F[i].piv.size() + F[c].piv.size()), m = p + double(F[i].border.size());
        if (m > kFrontMax) continue;
        const double base = F[i].work0 + F[c].work0, growth = (front_work(p, m) - base) / base;
        const bool small = p <= kSmallPivots && m <= kSmallRows && growth < kSmallGrowth;
        if ((small || growth < kGrowth) && (best < 0 || growth < best_growth)) {
          best = c;
          best_growth = growth;
        }
      }
      if (best < 0) break;
      Draft &C = F[best];
      C.piv.insert(C.piv.end(), F[i].piv.begin(), F[i].piv.end());
      F[i].piv.swap(C.piv);
      F[i].work0 += C.work0;
      F[i].child.erase(std::find(F[i].child.begin(), F[i].child.end(), best));
      for (int g : C.child) {
        F[g].parent = i;
        F[i].child.push_back(g);
      }
      C = Draft();
      C.gone = true;
    }
  }
}

}  // namespace

bool build_front_plan(const LuSymbolic &S, const int *rp, const int *ci, FrontPlan *plan) {
  FrontPlan &P = *plan;
  P = FrontPlan();
  const int n = P.n = S.n;
  for (int r = 0; r < n; ++r)
    for (int p = rp[r] + 1; p < rp[r + 1]; ++p)
      if (ci[p] <= ci[p - 1]) return false;
  std::vector<int> col_of;
  std::vector<char> kind_of;
  std::vector<std::vector<int>> first, last;
  if (!pair_rows(n, rp, ci, &col_of, &kind_of, &first, &last)) return false;
  P.Q.resize(n);
  std::vector<int> pinv(n);
  for (int k = 0; k < n; ++k) {
    P.Q[k] = col_of[S.P[k]];
    pinv[S.P[k]] = k;
  }
  for (auto *rounds : {&first, &last})
    for (auto &rows : *rounds)
      for (int &r : rows) r = pinv[r];
  std::vector<char> kind(n);
  for (int k = 0; k < n; ++k) kind[k] = kind_of[S.P[k]];
  const Matched B = match(n, S.P, P.Q, rp, ci);
  for (auto &r : first)
    add_round(P.before, B, std::move(r), true, [&](int c) { return kind[c] == BEFORE; });
  for (size_t k = last.size(); k-- > 0;)
    add_round(P.after, B, std::move(last[k]), true, [](int) { return true; });
  std::vector<int> core, place(n, -1);
  for (int k = 0; k < n; ++k)
    if (kind[k] == CORE) {
      place[k] = int(core.size());
      core.push_back(k);
    }
  const int nc = int(core.size());
  add_round(P.core, B, core, false, [&](int c) { return kind[c] == BEFORE; });
  if (nc == 0) return false;

  // order of the core
  Graph G;
  G.ptr.assign(1, 0);
  {
    std::vector<int> t;
    for (int a = 0; a < nc; ++a) {
      t.clear();
      const int k = core[a];
      for (int64_t q = B.rp[k]; q < B.rp[k + 1]; ++q)
        if (place[B.rcol[q]] >= 0 && B.rcol[q] != k) t.push_back(place[B.rcol[q]]);
      for (int64_t q = B.cp[k]; q < B.cp[k + 1]; ++q)
        if (place[B.crow[q]] >= 0 && B.crow[q] != k) t.push_back(place[B.crow[q]]);
      std::sort(t.begin(), t.end());
      t.erase(std::unique(t.begin(), t.end()), t.end());
      G.adj.insert(G.adj.end(), t.begin(), t.end());
      G.ptr.push_back(int(G.adj.size()));
    }
  }
  const std::vector<int> order = Dissection(G).order();
  std::vector<int> pos(nc);
  for (int k = 0; k < nc; ++k) pos[order[k]] = k;

  // symbolic elimination: the later positions column k touches
  std::vector<std::vector<int>> touch(nc), kids(nc);
  {
    std::vector<int> mark(nc, -1);
    for (int k = 0; k < nc; ++k) {
      std::vector<int> t;
      const int a = order[k];
      for (int e = G.ptr[a]; e < G.ptr[a + 1]; ++e) {
        const int j = pos[G.adj[e]];
        if (j > k && mark[j] != k) {
          mark[j] = k;
          t.push_back(j);
        }
      }
      for (int c : kids[k])
        for (int j : touch[c])
          if (j > k && mark[j] != k) {
            mark[j] = k;
            t.push_back(j);
          }
      if (int(t.size()) >= kFrontMax) return false;
      std::sort(t.begin(), t.end());
      if (!t.empty()) kids[t[0]].push_back(k);
      touch[k] = std::move(t);
    }
  }
  // columns with the same border as their only child's share its front
  std::vector<Draft> F;
  {
    std::vector<int> front_of(nc, -1);
    for (int k = 0; k < nc; ++k) {
      const int c = kids[k].size() == 1 ? kids[k][0] : -1;
      if (c >= 0 && touch[c].size() == touch[k].size() + 1 && F[front_of[c]].piv.size() + touch[c].size() < kFrontMax) {
        front_of[k] = front_of[c];
      } else {
        front_of[k] = int(F.size());
        F.emplace_back();
      }
      F[front_of[k]].piv.push_back(k);
      F[front_of[k]].border = touch[k];
    }
    for (size_t i = 0; i < F.size(); ++i) {
      F[i].work0 = front_work(double(F[i].piv.size()), double(F[i].piv.size() + F[i].border.size()));
      if (F[i].border.empty()) continue;
      F[i].parent = front_of[F[i].border[0]];
      F[F[i].parent].child.push_back(int(i));
    }
    std::vector<std::vector<int>>().swap(touch);
    std::vector<int> by_pivot(F.size());
    std::iota(by_pivot.begin(), by_pivot.end(), 0);
    std::sort(by_pivot.begin(), by_pivot.end(), [&](int a, int b) { return F[a].piv.back() < F[b].piv.back(); });
    merge_fronts(F, by_pivot);
    for (int i : by_pivot) {
      if (F[i].gone || F[i].parent < 0) continue;
      Draft &U = F[F[i].parent];
      U.level = std::max(U.level, F[i].level + 1);
    }
  }
  // fronts by level, size class and work
  std::vector<int> seq;
  int top = 0;
  for (size_t i = 0; i < F.size(); ++i)
    if (!F[i].gone) {
      seq.push_back(int(i));
      top = std::max(top, F[i].level);
      if (F[i].child.size() > size_t(kFrontMaxChildren)) return false;
    }
  auto rows_of = [&](int i) { return int(F[i].piv.size() + F[i].border.size()); };
  auto class_of = [&](int i) { return rows_of(i) > kFrontMiddle ? 0 : rows_of(i) > kFrontLow ? 1 : 2; };
  auto work_of = [&](int i) { return front_work(double(F[i].piv.size()), rows_of(i)); };
  std::stable_sort(seq.begin(), seq.end(), [&](int a, int b) {
    if (F[a].level != F[b].level) return F[a].level < F[b].level;
    if (class_of(a) != class_of(b)) return class_of(a) < class_of(b);
    return work_of(a) > work_of(b);
  });
  std::vector<int> number(F.size(), -1);
  for (size_t k = 0; k < seq.size(); ++k) number[seq[k]] = int(k);
  P.level.assign(top + 2, 0);
  for (int i : seq) ++P.level[F[i].level + 1];
  for (int l = 0; l <= top; ++l) P.level[l + 1] += P.level[l];

  // the merged fronts' elimination order: a column's place decides which of
  // two fronts an entry of A belongs to
  std::vector<int> owner(nc, -1), rank(nc, -1);  // by position: front, place among its pivots
  for (int i : seq)
    for (size_t k = 0; k < F[i].piv.size(); ++k) {
      owner[F[i].piv[k]] = number[i];
      rank[F[i].piv[k]] = int(k);
    }
  P.front.resize(seq.size());
  std::vector<int> local(nc, -1);
  for (size_t s = 0; s < seq.size(); ++s) {
    const Draft &D = F[seq[s]];
    Front &f = P.front[s];
    f.p = int(D.piv.size());
    f.m = f.p + int(D.border.size());
    f.level = D.level;
    f.parent = D.parent >= 0 ? number[D.parent] : -1;
    f.idx = int64_t(P.idx.size());
    const int64_t b = f.m - f.p;
    f.lo = P.n_l;
    f.uo = P.n_u;
    f.co = P.n_c;
    f.pv = P.n_pv;
    f.bv = P.n_bv;
    P.n_l += int64_t(f.m) * f.p;
    P.n_u += b * f.p;
    P.n_c += b * b;
    P.n_pv += f.p;
    P.n_bv += b;
    P.flops += front_work(f.p, f.m);
    for (int k : D.piv) P.idx.push_back(core[order[k]]);
    for (int k : D.border) P.idx.push_back(core[order[k]]);
    // children, in the order of their numbers, and the places of their borders
    for (int k = 0; k < f.p; ++k) local[D.piv[k]] = k;
    for (int k = 0; k < int(b); ++k) local[D.border[k]] = f.p + k;
    std::vector<int> kids_of;
    for (int c : D.child) kids_of.push_back(c);
    std::sort(kids_of.begin(), kids_of.end(), [&](int x, int y) { return number[x] < number[y]; });
    f.child0 = int(P.child.size());
    for (int c : kids_of) {
      P.child.push_back(number[c]);
      P.inv.push_back(int64_t(P.inv_map.size()));
      P.inv_map.resize(P.inv_map.size() + size_t(f.m), -1);
      int *inv = P.inv_map.data() + P.inv.back();
      P.front[number[c]].map = int64_t(P.map.size());
      for (size_t k = 0; k < F[c].border.size(); ++k) {
        const int at = local[F[c].border[k]];
        P.map.push_back(at);
        inv[at] = int(k);
      }
    }
    f.child1 = int(P.child.size());
    // A entries with their first index among the pivots, by column
    std::vector<std::vector<std::pair<int, int>>> cols(f.m);
    auto later = [&](int j, int k) {  // position j is eliminated with or after pivot k of this front
      return owner[j] != int(s) || rank[j] >= k;
    };
    for (int k = 0; k < f.p; ++k) {
      const int row = core[order[D.piv[k]]];
      for (int64_t q = B.rp[row]; q < B.rp[row + 1]; ++q) {
        const int c = place[B.rcol[q]];
        if (c < 0) continue;
        const int j = pos[c];
        if (local[j] >= 0 && later(j, k)) cols[local[j]].push_back({k, B.ra[q]});
      }
      for (int64_t q = B.cp[row]; q < B.cp[row + 1]; ++q) {
        const int r = place[B.crow[q]];
        if (r < 0 || B.crow[q] == row) continue;
        const int j = pos[r];
        if (local[j] >= 0 && later(j, k + 1)) cols[k].push_back({local[j], B.ca[q]});
      }
    }
    f.acol = int64_t(P.apos.size());
    for (int j = 0; j < f.m; ++j)
      for (auto &e : cols[j]) {
        P.apos.push_back(j * kFrontMax + e.first);
        P.aidx.push_back(e.second);
      }
    f.na = int(int64_t(P.apos.size()) - f.acol);
    for (int k : D.piv) local[k] = -1;
    for (int k : D.border) local[k] = -1;
  }
  // modelled time: a level waits for its longest front (launch and assembly,
  // its pivots in turn, its work on the SMs it can take) and for its share of
  // the chip's FP64 rate (power grids of 668 to 120,002 rows and logic blocks
  // of 3,000 to 200,000 devices take 0.78 to 1.03 times it, chains of 2,000 and
  // 7,000 stages 0.7)
  for (int l = 0; l <= top; ++l) {
    double total = 0, longest = 0, pivots = 0;
    for (int k = P.level[l]; k < P.level[l + 1]; ++k) {
      total += front_work(P.front[k].p, P.front[k].m);
      longest = std::max(longest, front_work(P.front[k].p, P.front[k].m));
      pivots = std::max(pivots, double(P.front[k].p));
    }
    const double sms = std::min(16.0, std::max(1.0, kModelSms / (P.level[l + 1] - P.level[l])));
    P.seconds += 20e-6 + pivots * 1.1e-6 + std::max(longest / (sms * 4e9), total / 600e9);
  }
  return true;
}

}  // namespace xg
