// Nested-dissection ordering and multifrontal symbolic factorisation on the
// host.  The numeric work happens on the GPU (mf_kernels.cu).
#include "mf_symbolic.hpp"

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <stdexcept>
#include <thread>

namespace dg {
namespace {

struct Graph {  // symmetric adjacency without self loops
  int n = 0;
  std::vector<int64_t> ptr;
  std::vector<int> adj;
};

// One matrix' symbolic result before it is placed into the batch.
struct Local {
  int n = 0;
  std::vector<int> perm;      // new -> local
  std::vector<int> iperm;     // local -> new
  // fronts in creation (post) order
  std::vector<int> p0, k, parent, level;
  std::vector<std::vector<int>> children;
  std::vector<std::vector<int>> rows;  // pivots then update rows (new numbering)
  // lower-triangle entries: (new row, new col, source index)
  std::vector<int> er, ec;
  std::vector<int64_t> es;
};

class Dissector {
 public:
  Dissector(const Graph &g, int leaf, Local &L) : g_(g), leaf_(leaf), L_(L) {
    mark_.assign((size_t)g.n, 0);
    lev_.assign((size_t)g.n, -1);
  }

  void run() {
    std::vector<int> all((size_t)g_.n);
    for (int i = 0; i < g_.n; i++) all[(size_t)i] = i;
    std::vector<int> roots;
    dissect(all, roots);
  }

 private:
  // BFS restricted to the set stamped with `stamp`; returns visit order and
  // fills lev_ for visited nodes.
  void bfs(int s, int stamp, std::vector<int> &order, int &nlev) {
    order.clear();
    order.push_back(s);
    lev_[(size_t)s] = 0;
    mark_[(size_t)s] = -stamp;
    nlev = 1;
    for (size_t h = 0; h < order.size(); h++) {
      int v = order[h];
      for (int64_t e = g_.ptr[(size_t)v]; e < g_.ptr[(size_t)v + 1]; e++) {
        int w = g_.adj[(size_t)e];
        if (mark_[(size_t)w] == stamp) {
          mark_[(size_t)w] = -stamp;
          lev_[(size_t)w] = lev_[(size_t)v] + 1;
          nlev = std::max(nlev, lev_[(size_t)w] + 1);
          order.push_back(w);
        }
      }
    }
    for (int v : order) mark_[(size_t)v] = stamp;  // restore membership
  }

  int new_front(const std::vector<int> &piv) {
    int f = (int)L_.p0.size();
    L_.p0.push_back((int)L_.perm.size());
    L_.k.push_back((int)piv.size());
    L_.parent.push_back(-1);
    L_.level.push_back(0);
    L_.children.emplace_back();
    for (int v : piv) L_.perm.push_back(v);
    return f;
  }

  void dissect(std::vector<int> &nodes, std::vector<int> &roots) {
    roots.clear();
    if (nodes.empty()) return;
    int stamp = ++stamp_;
    for (int v : nodes) mark_[(size_t)v] = stamp;
    // connected components
    std::vector<int> order;
    std::vector<std::vector<int>> comps;
    {
      int cstamp = ++stamp_;
      (void)cstamp;
      std::vector<char> seen;
      for (int v : nodes) {
        if (mark_[(size_t)v] != stamp) continue;  // already taken by a component
        int nl;
        bfs(v, stamp, order, nl);
        for (int w : order) mark_[(size_t)w] = 0;  // remove from the pending set
        comps.push_back(order);
      }
    }
    if (comps.size() > 1) {
      // components larger than a leaf are dissected on their own; the small
      // ones are packed together into leaf fronts (one dense front may hold
      // several disconnected pieces), which keeps tiny fronts with large
      // boundaries out of the tree
      std::vector<int> pack;
      auto flush = [&]() {
        if (!pack.empty()) { roots.push_back(new_front(pack)); pack.clear(); }
      };
      for (auto &c : comps) {
        if ((int)c.size() > leaf_) {
          std::vector<int> r;
          dissect(c, r);
          roots.insert(roots.end(), r.begin(), r.end());
        } else {
          if ((int)(pack.size() + c.size()) > leaf_) flush();
          pack.insert(pack.end(), c.begin(), c.end());
        }
      }
      flush();
      return;
    }
    std::vector<int> &S = comps[0];
    int N = (int)S.size();
    if (N <= leaf_) {
      roots.push_back(new_front(S));
      return;
    }
    stamp = ++stamp_;
    for (int v : S) mark_[(size_t)v] = stamp;
    // pseudo-peripheral start: two sweeps
    int nl = 0;
    bfs(S[0], stamp, order, nl);
    int s = order.back();
    bfs(s, stamp, order, nl);
    s = order.back();
    bfs(s, stamp, order, nl);
    if (nl < 3) {
      for (int v : S) mark_[(size_t)v] = 0;
      roots.push_back(new_front(S));
      return;
    }
    std::vector<int> cnt((size_t)nl, 0);
    for (int v : order) cnt[(size_t)lev_[(size_t)v]]++;
    // separator: a level near the middle with few nodes
    int best = -1;
    int64_t before = 0;
    double bestscore = 1e300;
    for (int l = 0; l < nl; l++) {
      int64_t after = N - before - cnt[(size_t)l];
      if (l > 0 && l < nl - 1) {
        double bal = std::fabs((double)before - (double)after) / (double)N;
        if (before >= (int64_t)(0.25 * N) && after >= (int64_t)(0.25 * N)) {
          double score = (double)cnt[(size_t)l] * (1.0 + bal);
          if (score < bestscore) { bestscore = score; best = l; }
        }
      }
      before += cnt[(size_t)l];
    }
    if (best < 0) {  // fall back to the median level
      before = 0;
      for (int l = 0; l < nl; l++) {
        if (before + cnt[(size_t)l] >= N / 2) { best = std::min(std::max(l, 1), nl - 2); break; }
        before += cnt[(size_t)l];
      }
    }
    std::vector<int> A, B, Sep;
    for (int v : order) {
      int l = lev_[(size_t)v];
      if (l < best) A.push_back(v);
      else if (l > best) B.push_back(v);
      else Sep.push_back(v);
    }
    for (int v : S) mark_[(size_t)v] = 0;
    std::vector<int> ra, rb;
    dissect(A, ra);
    dissect(B, rb);
    int f = new_front(Sep);
    for (int c : ra) { L_.children[(size_t)f].push_back(c); L_.parent[(size_t)c] = f; }
    for (int c : rb) { L_.children[(size_t)f].push_back(c); L_.parent[(size_t)c] = f; }
    roots.push_back(f);
  }

  const Graph &g_;
  int leaf_;
  Local &L_;
  std::vector<int> mark_, lev_;
  int stamp_ = 0;
};

// Front row structure: pivots, then the later-numbered rows adjacent to the
// front's subtree (the multifrontal update rows).
void finish_local(const Graph &g, Local &L) {
  int n = g.n;
  L.iperm.assign((size_t)n, 0);
  for (int i = 0; i < n; i++) L.iperm[(size_t)L.perm[(size_t)i]] = i;
  int nf = (int)L.p0.size();
  L.rows.assign((size_t)nf, {});
  std::vector<int> stamp((size_t)n, -1);
  for (int f = 0; f < nf; f++) {  // creation order is a post-order
    int p0 = L.p0[(size_t)f], k = L.k[(size_t)f], last = p0 + k - 1;
    std::vector<int> U;
    for (int q = 0; q < k; q++) {
      int v = L.perm[(size_t)(p0 + q)];
      for (int64_t e = g.ptr[(size_t)v]; e < g.ptr[(size_t)v + 1]; e++) {
        int w = L.iperm[(size_t)g.adj[(size_t)e]];
        if (w > last && stamp[(size_t)w] != f) { stamp[(size_t)w] = f; U.push_back(w); }
      }
    }
    int lev = 0;
    for (int c : L.children[(size_t)f]) {
      const std::vector<int> &rc = L.rows[(size_t)c];
      for (size_t q = (size_t)L.k[(size_t)c]; q < rc.size(); q++) {
        int w = rc[q];
        if (w > last && stamp[(size_t)w] != f) { stamp[(size_t)w] = f; U.push_back(w); }
      }
      lev = std::max(lev, L.level[(size_t)c] + 1);
    }
    L.level[(size_t)f] = L.children[(size_t)f].empty() ? 0 : lev;
    std::sort(U.begin(), U.end());
    std::vector<int> &R = L.rows[(size_t)f];
    R.reserve((size_t)k + U.size());
    for (int q = 0; q < k; q++) R.push_back(p0 + q);
    R.insert(R.end(), U.begin(), U.end());
  }
}

Graph graph_of_local(int n, const std::vector<int> &er, const std::vector<int> &ec) {
  Graph g;
  g.n = n;
  std::vector<int64_t> deg((size_t)n + 1, 0);
  for (size_t q = 0; q < er.size(); q++)
    if (er[q] != ec[q]) { deg[(size_t)er[q] + 1]++; deg[(size_t)ec[q] + 1]++; }
  for (int i = 0; i < n; i++) deg[(size_t)i + 1] += deg[(size_t)i];
  g.ptr = deg;
  std::vector<int> adj((size_t)deg[(size_t)n]);
  std::vector<int64_t> fill(deg.begin(), deg.end() - 1);
  for (size_t q = 0; q < er.size(); q++)
    if (er[q] != ec[q]) {
      adj[(size_t)fill[(size_t)er[q]]++] = ec[q];
      adj[(size_t)fill[(size_t)ec[q]]++] = er[q];
    }
  // dedupe
  g.ptr.assign((size_t)n + 1, 0);
  std::vector<int> mark((size_t)n, -1);
  g.adj.clear();
  g.adj.reserve(adj.size());
  for (int i = 0; i < n; i++) {
    for (int64_t e = deg[(size_t)i]; e < deg[(size_t)i + 1]; e++) {
      int w = adj[(size_t)e];
      if (mark[(size_t)w] != i) { mark[(size_t)w] = i; g.adj.push_back(w); }
    }
    g.ptr[(size_t)i + 1] = (int64_t)g.adj.size();
  }
  return g;
}

// One matrix between its dissection and its placement: the graph and the
// fronts of the dissection tree.
struct Work {
  Graph g;
  Local L;
  std::vector<int> gid, lr, lc;
  std::vector<int64_t> src;
};

void dissect(Work &w, int n, int leaf) {
  w.g = graph_of_local(n, w.lr, w.lc);
  w.L = Local();
  w.L.n = n;
  Dissector d(w.g, leaf, w.L);
  d.run();
  finish_local(w.g, w.L);
}

// Joining levels.  A level costs at least a launch and a chain of loads
// however little it holds, so a short one is better joined with the next:
// consecutive levels become one, in which a front takes its descendants of
// those levels in (their pivots first, then its own; its update rows stay).
// Its elimination matrix holds more entries than theirs together (siblings
// are not coupled), and its factorisation walks their pivots one after the
// other.
constexpr int kJoin = 4;  // levels joined at most

// Of the level that the levels h .. h + g make, per h and g: entries of the
// elimination matrices, multiply-adds of the factorisation, the most pivots
// and rows of a front, fronts.
struct LevelSums {
  double entries[kJoin] = {}, work[kJoin] = {}, pivots[kJoin] = {}, rows[kJoin] = {};
  int fronts[kJoin] = {};
};

void add_sums(const Local &L, std::vector<LevelSums> &out) {
  const int nf = (int)L.p0.size();
  std::vector<double> kk((size_t)nf * kJoin);  // pivots of f and its descendants of up to j levels below
  for (int f = 0; f < nf; f++) {               // children come first
    const int H = L.level[(size_t)f], up = L.parent[(size_t)f];
    const int Hp = up < 0 ? 1 << 30 : L.level[(size_t)up];
    const double r = (double)L.rows[(size_t)f].size() - L.k[(size_t)f];
    if ((int)out.size() <= H) out.resize((size_t)H + 1);
    for (int j = 0; j < kJoin && j <= H; j++) {
      double k = L.k[(size_t)f];
      for (int c : L.children[(size_t)f]) {
        const int jc = L.level[(size_t)c] - (H - j);
        if (jc >= 0) k += kk[(size_t)c * kJoin + jc];
      }
      kk[(size_t)f * kJoin + j] = k;
      LevelSums &S = out[(size_t)(H - j)];
      for (int g = j; g < kJoin && H - j + g < Hp; g++) {  // f is the top front of its group
        S.entries[g] += k * (k + r) - 0.5 * k * k;
        S.work[g] += k * (k * k / 3 + r * k + r * r) / 2;
        S.pivots[g] = std::max(S.pivots[g], k);
        S.rows[g] = std::max(S.rows[g], k + r);
        S.fronts[g]++;
      }
    }
  }
}

// Group of each level: the cheapest split of the levels for a factorisation
// and kNominal solves.  In microseconds, per level: both directions of a solve
// 4.5 and the entries at the rate of short levels (FP64 250, FP32 500 per ns);
// the factorisation 35 for the assembly, 37 per 32 pivots of the longest
// front, 2 multiply-adds per ps.  A level of opt.thin fronts and more is not
// joined: its fronts are solved by groups of lanes that walk the pivots.
// Launches and time per iteration without and with: Poisson 129^2 48 and 22,
// 141 and 87 us; diffusion 45^3 43 and 24, 330 and 284 us; elasticity 26^3 mixed
// 36 and 23, 155 and 127 us; 128^3 mixed, whose lower levels are long, 71 and 59,
// 1145 and 1116 us.  FP32 at 300 per ns joins too little (elasticity 138 us), at
// 1200 too much where several right-hand sides share a level (32 of 513^2: 1591 us
// against 1518).
std::vector<int> plan_joins(const std::vector<LevelSums> &S, const MfOptions &opt) {
  const int N = (int)S.size();
  constexpr double kNominal = 30;
  const double rate = opt.value_bytes == 8 ? 250e3 : 500e3;
  std::vector<double> best((size_t)N + 1, 0.0);
  std::vector<int> len((size_t)N + 1, 1);
  for (int h = N - 1; h >= 0; h--) {
    best[(size_t)h] = 1e300;
    for (int g = 0; g < kJoin && h + g < N; g++) {
      const LevelSums &s = S[(size_t)h];
      if (g > 0 && (s.fronts[g] >= opt.thin || s.rows[g] > opt.max_rows)) continue;
      const double t = 2 * kNominal * (4.5 + s.entries[g] / rate) + 35 + 37 * std::ceil(s.pivots[g] / 32) +
                       s.work[g] / 2e6 + best[(size_t)(h + g + 1)];
      if (t < best[(size_t)h]) { best[(size_t)h] = t; len[(size_t)h] = g + 1; }
    }
  }
  std::vector<int> group((size_t)N);
  for (int h = 0; h < N; h += len[(size_t)h])
    for (int q = h; q < std::min(N, h + len[(size_t)h]); q++) group[(size_t)q] = h;
  return group;
}

void join(Work &w, const std::vector<int> &group) {
  const Local &O = w.L;
  const int nf = (int)O.p0.size();
  std::vector<int> top((size_t)nf), id((size_t)nf, -1);  // the front that takes f in; its new number
  bool any = false;
  for (int f = nf - 1; f >= 0; f--) {  // parents first
    const int up = O.parent[(size_t)f];
    const bool in = up >= 0 && group[(size_t)O.level[(size_t)f]] == group[(size_t)O.level[(size_t)up]];
    top[(size_t)f] = in ? top[(size_t)up] : f;
    any |= in;
  }
  if (!any) return;
  Local L;
  L.n = O.n;
  std::vector<std::vector<int>> members((size_t)nf);
  for (int f = 0; f < nf; f++) members[(size_t)top[(size_t)f]].push_back(f);  // post-order
  for (int f = 0; f < nf; f++) {
    if (top[(size_t)f] != f) continue;
    const int id_f = (int)L.p0.size();
    id[(size_t)f] = id_f;
    L.p0.push_back((int)L.perm.size());
    L.parent.push_back(-1);
    L.level.push_back(0);
    L.children.emplace_back();
    int k = 0;
    for (int q : members[(size_t)f]) {
      for (int i = 0; i < O.k[(size_t)q]; i++) L.perm.push_back(O.perm[(size_t)(O.p0[(size_t)q] + i)]);
      k += O.k[(size_t)q];
      for (int c : O.children[(size_t)q])
        if (top[(size_t)c] == c) {
          L.children.back().push_back(id[(size_t)c]);
          L.parent[(size_t)id[(size_t)c]] = id_f;
        }
    }
    L.k.push_back(k);
  }
  w.L = std::move(L);
  finish_local(w.g, w.L);
}

// the entries of the lower triangle in the new numbering
void place_entries(Work &w) {
  Local &L = w.L;
  const std::vector<int> &lr = w.lr, &lc = w.lc;
  const std::vector<int64_t> &src = w.src;
  // keep entries of the lower triangle in the new numbering
  for (size_t q = 0; q < lr.size(); q++) {
    int a = L.iperm[(size_t)lr[q]], b = L.iperm[(size_t)lc[q]];
    if (a >= b) { L.er.push_back(a); L.ec.push_back(b); L.es.push_back(src[q]); }
  }
}

void append(const Local &L, const std::vector<int> &gid_of_local, MfBatch &B) {
  int base_front = B.nfronts;
  int64_t xoff = B.xlen;
  B.xoff.push_back(xoff);
  for (int i = 0; i < L.n; i++) B.gidx.push_back(gid_of_local[(size_t)L.perm[(size_t)i]]);
  B.xlen += L.n;
  int nf = (int)L.p0.size();
  // owner front of each pivot
  std::vector<int> owner((size_t)L.n, -1);
  for (int f = 0; f < nf; f++)
    for (int q = 0; q < L.k[(size_t)f]; q++) owner[(size_t)(L.p0[(size_t)f] + q)] = f;
  std::vector<int64_t> foff((size_t)nf);
  for (int f = 0; f < nf; f++) {
    int m = (int)L.rows[(size_t)f].size(), k = L.k[(size_t)f];
    foff[(size_t)f] = B.arena;
    B.f_off.push_back(B.arena);
    B.arena += ((int64_t)m * m + 3) & ~(int64_t)3;  // 16-byte aligned fronts (cp.async staging)
    B.f_m.push_back(m);
    B.f_k.push_back(k);
    B.f_rows.push_back((int64_t)B.rows.size());
    B.rows.insert(B.rows.end(), L.rows[(size_t)f].begin(), L.rows[(size_t)f].end());
    B.f_xoff.push_back(xoff);
    B.f_p0.push_back(L.p0[(size_t)f]);
    B.f_uoff.push_back(B.ulen);
    B.ulen += m - k;
    B.f_woff.push_back(B.wlen);
    B.wlen += m;
    B.f_parent.push_back(L.parent[(size_t)f] < 0 ? -1 : L.parent[(size_t)f] + base_front);
    B.f_level.push_back(L.level[(size_t)f]);
    B.factor_nnz += (int64_t)m * k - (int64_t)k * (k - 1) / 2;
    double r = m - k;
    B.factor_flops += (double)k * k * k / 3.0 + r * k * k + r * r * k;
    B.max_m = std::max(B.max_m, m);
  }
  for (int f = 0; f < nf; f++) {
    B.f_child_ptr.push_back((int)B.f_children.size());
    for (int c : L.children[(size_t)f]) B.f_children.push_back(c + base_front);
  }
  // relmaps: child update rows -> positions in the parent's row list
  for (int f = 0; f < nf; f++) {
    B.f_relmap.push_back((int64_t)B.relmap.size());
    int p = L.parent[(size_t)f];
    const std::vector<int> &rc = L.rows[(size_t)f];
    int k = L.k[(size_t)f];
    if (p < 0) {
      if ((int)rc.size() != k) throw std::runtime_error("root front with update rows");
      continue;
    }
    const std::vector<int> &rp = L.rows[(size_t)p];
    for (size_t q = (size_t)k; q < rc.size(); q++) {
      auto it = std::lower_bound(rp.begin(), rp.end(), rc[q]);
      if (it == rp.end() || *it != rc[q]) throw std::runtime_error("update row missing in parent");
      B.relmap.push_back((int)(it - rp.begin()));
    }
  }
  // assembly entries, grouped by target (duplicates summed in entry order)
  std::vector<std::pair<int64_t, int64_t>> te;  // (target, source)
  te.reserve(L.er.size());
  for (size_t q = 0; q < L.er.size(); q++) {
    int a = L.er[q], b = L.ec[q];
    int f = owner[(size_t)b];
    const std::vector<int> &R = L.rows[(size_t)f];
    auto it = std::lower_bound(R.begin(), R.end(), a);
    if (it == R.end() || *it != a) throw std::runtime_error("entry row not in its front");
    int64_t row = it - R.begin();
    int64_t col = b - L.p0[(size_t)f];
    int64_t m = (int64_t)R.size();
    te.emplace_back(foff[(size_t)f] + col * m + row, L.es[q]);
  }
  std::stable_sort(te.begin(), te.end(),
                   [](const std::pair<int64_t, int64_t> &x, const std::pair<int64_t, int64_t> &y) {
                     return x.first < y.first;
                   });
  // per-front entry ranges (entries are sorted by target, fronts by offset)
  {
    size_t e = 0;
    int64_t ent = (int64_t)B.asm_tgt.size();
    for (int ff = 0; ff < nf; ff++) {
      B.f_asm.push_back(ent);
      int64_t end = foff[(size_t)ff] + (int64_t)L.rows[(size_t)ff].size() * L.rows[(size_t)ff].size();
      while (e < te.size() && te[e].first < end) {
        int64_t t = te[e].first;
        B.asm_tgt.push_back(t);
        B.asm_sp.push_back((int64_t)B.asm_src.size());
        while (e < te.size() && te[e].first == t) { B.asm_src.push_back(te[e].second); e++; }
        ent++;
      }
    }
  }
  B.nmat++;
  B.nfronts += nf;
}

// Appends batch P (built by append from an empty batch) to B: the result is
// what appending P's matrices to B directly gives (offsets shifted by B's
// sizes; the flop count is summed per piece).
void merge(const MfBatch &P, MfBatch &B) {
  const int base_front = B.nfronts;
  const int64_t arena = B.arena, xlen = B.xlen, ulen = B.ulen, wlen = B.wlen;
  const int64_t nrows = (int64_t)B.rows.size(), nrel = (int64_t)B.relmap.size();
  const int64_t nasm = (int64_t)B.asm_tgt.size(), nsrc = (int64_t)B.asm_src.size();
  const int nchild = (int)B.f_children.size();
  for (int64_t v : P.xoff) B.xoff.push_back(v + xlen);
  B.gidx.insert(B.gidx.end(), P.gidx.begin(), P.gidx.end());
  for (int64_t v : P.f_off) B.f_off.push_back(v + arena);
  B.f_m.insert(B.f_m.end(), P.f_m.begin(), P.f_m.end());
  B.f_k.insert(B.f_k.end(), P.f_k.begin(), P.f_k.end());
  for (int64_t v : P.f_rows) B.f_rows.push_back(v + nrows);
  for (int64_t v : P.f_xoff) B.f_xoff.push_back(v + xlen);
  B.f_p0.insert(B.f_p0.end(), P.f_p0.begin(), P.f_p0.end());
  for (int64_t v : P.f_uoff) B.f_uoff.push_back(v + ulen);
  for (int64_t v : P.f_woff) B.f_woff.push_back(v + wlen);
  for (int v : P.f_child_ptr) B.f_child_ptr.push_back(v + nchild);
  for (int v : P.f_children) B.f_children.push_back(v + base_front);
  for (int64_t v : P.f_relmap) B.f_relmap.push_back(v + nrel);
  for (int64_t v : P.f_asm) B.f_asm.push_back(v + nasm);
  for (int v : P.f_parent) B.f_parent.push_back(v < 0 ? -1 : v + base_front);
  B.f_level.insert(B.f_level.end(), P.f_level.begin(), P.f_level.end());
  B.rows.insert(B.rows.end(), P.rows.begin(), P.rows.end());
  B.relmap.insert(B.relmap.end(), P.relmap.begin(), P.relmap.end());
  for (int64_t v : P.asm_tgt) B.asm_tgt.push_back(v + arena);
  for (int64_t v : P.asm_sp) B.asm_sp.push_back(v + nsrc);
  B.asm_src.insert(B.asm_src.end(), P.asm_src.begin(), P.asm_src.end());
  B.nmat += P.nmat;
  B.nfronts += P.nfronts;
  B.arena += P.arena;
  B.xlen += P.xlen;
  B.ulen += P.ulen;
  B.wlen += P.wlen;
  B.factor_nnz += P.factor_nnz;
  B.factor_flops += P.factor_flops;
  B.max_m = std::max(B.max_m, P.max_m);
}

void finalize(MfBatch &B) {
  B.xoff.push_back(B.xlen);
  B.arena += 16;  // slack: staging copies round the last front up to 16 bytes
  B.f_child_ptr.push_back((int)B.f_children.size());
  B.f_asm.push_back((int64_t)B.asm_tgt.size());
  B.asm_sp.push_back((int64_t)B.asm_src.size());
  int L = 0;
  for (int lv : B.f_level) L = std::max(L, lv + 1);
  B.nlevels = L;
  B.lvl_ptr.assign((size_t)L + 1, 0);
  for (int lv : B.f_level) B.lvl_ptr[(size_t)lv + 1]++;
  for (int l = 0; l < L; l++) B.lvl_ptr[(size_t)l + 1] += B.lvl_ptr[(size_t)l];
  B.lvl_fronts.assign((size_t)B.nfronts, 0);
  std::vector<int> fill(B.lvl_ptr.begin(), B.lvl_ptr.end() - 1);
  for (int f = 0; f < B.nfronts; f++) B.lvl_fronts[(size_t)fill[(size_t)B.f_level[(size_t)f]]++] = f;
  // largest fronts first inside a level, so that long blocks start early
  for (int l = 0; l < L; l++)
    std::stable_sort(B.lvl_fronts.begin() + B.lvl_ptr[(size_t)l], B.lvl_fronts.begin() + B.lvl_ptr[(size_t)l + 1],
                     [&](int a, int b) { return B.f_m[(size_t)a] > B.f_m[(size_t)b]; });
  B.lvl_max_m.assign((size_t)L, 0);
  for (int l = 0; l < L; l++)
    for (int q = B.lvl_ptr[(size_t)l]; q < B.lvl_ptr[(size_t)l + 1]; q++)
      B.lvl_max_m[(size_t)l] = std::max(B.lvl_max_m[(size_t)l], B.f_m[(size_t)B.lvl_fronts[(size_t)q]]);
}

// Nodes of a subdomain are looked up by an array over their range up to this
// many times the subdomain's size (128 bytes a node on each host thread).
constexpr int64_t kLookupRange = 32;

template <class F>
void parallel_for(int n, F fn) {
  unsigned nt = std::max(1u, std::min({std::thread::hardware_concurrency(), 32u, (unsigned)std::max(n, 1)}));
  if (n < 2 || nt < 2) {
    for (int i = 0; i < n; i++) fn(i);
    return;
  }
  std::atomic<int> next{0};
  std::vector<std::thread> th;
  for (unsigned t = 0; t < nt; t++)
    th.emplace_back([&] {
      for (;;) {
        int i = next.fetch_add(1);
        if (i >= n) break;
        fn(i);
      }
    });
  for (auto &t : th) t.join();
}

}  // namespace

void mf_build_subdomains(const Csr &A, const std::vector<int64_t> &sd_ptr,
                         const std::vector<int> &sd_nodes, const MfOptions &opt, MfBatch &out) {
  out = MfBatch();
  int nsd = (int)sd_ptr.size() - 1;
  // every subdomain is analysed and laid out as its own batch on a host
  // thread; the pieces are then joined in subdomain order
  std::vector<MfBatch> pieces((size_t)nsd);
  std::vector<Work> work((size_t)nsd);
  parallel_for(nsd, [&](int s) {
    int64_t b0 = sd_ptr[(size_t)s], m = sd_ptr[(size_t)s + 1] - b0;
    std::vector<int> &gid = work[(size_t)s].gid;
    gid.resize((size_t)m);
    // local position of each global node: an array over the subdomain's range
    // of nodes, or, where that is many times the subdomain, a sorted list (both
    // keep memory per subdomain small)
    int lo = INT_MAX, hi = -1;
    for (int64_t t = 0; t < m; t++) {
      const int g = gid[(size_t)t] = sd_nodes[(size_t)(b0 + t)] - 1;
      lo = std::min(lo, g);
      hi = std::max(hi, g);
    }
    const bool dense = (int64_t)hi - lo < kLookupRange * m;
    std::vector<int> pos;
    std::vector<std::pair<int, int>> lut;
    if (dense) {
      pos.assign((size_t)(hi - lo + 1), -1);
      for (int64_t t = m - 1; t >= 0; t--) pos[(size_t)(gid[(size_t)t] - lo)] = (int)t;
    } else {
      lut.resize((size_t)m);
      for (int64_t t = 0; t < m; t++) lut[(size_t)t] = {gid[(size_t)t], (int)t};
      std::sort(lut.begin(), lut.end());
    }
    auto loc = [&](int g) -> int {
      if (dense) return g < lo || g > hi ? -1 : pos[(size_t)(g - lo)];
      auto it = std::lower_bound(lut.begin(), lut.end(), std::make_pair(g, -1));
      if (it != lut.end() && it->first == g) return it->second;
      return -1;
    };
    int64_t most = 0;  // entries of the subdomain's rows
    for (int64_t t = 0; t < m; t++) most += A.ptr[(size_t)gid[(size_t)t] + 1] - A.ptr[(size_t)gid[(size_t)t]];
    std::vector<int> &lr = work[(size_t)s].lr, &lc = work[(size_t)s].lc;
    std::vector<int64_t> &src = work[(size_t)s].src;
    lr.reserve((size_t)most); lc.reserve((size_t)most); src.reserve((size_t)most);
    for (int64_t t = 0; t < m; t++) {
      int g = gid[(size_t)t];
      for (int64_t e = A.ptr[(size_t)g]; e < A.ptr[(size_t)g + 1]; e++) {
        int h = loc(A.col[(size_t)e]);
        if (h >= 0) { lr.push_back((int)t); lc.push_back(h); src.push_back(e); }
      }
    }
    dissect(work[(size_t)s], (int)m, opt.leaf);
  });
  std::vector<int> group;
  {
    std::vector<LevelSums> sums;
    for (const Work &w : work) add_sums(w.L, sums);
    group = plan_joins(sums, opt);
  }
  parallel_for(nsd, [&](int s) {
    Work &w = work[(size_t)s];
    join(w, group);
    place_entries(w);
    std::vector<int>().swap(w.lr);
    std::vector<int>().swap(w.lc);
    std::vector<int64_t>().swap(w.src);
    append(w.L, w.gid, pieces[(size_t)s]);
    w = Work();
  });
  // reserve the batch arrays once (they are large for big subdomains)
  {
    size_t nf = 0, nr = 0, ne = 0, nsrc = 0, nx = 0;
    for (const MfBatch &P : pieces) {
      nf += (size_t)P.nfronts;
      nr += P.rows.size();
      ne += P.asm_tgt.size();
      nsrc += P.asm_src.size();
      nx += P.gidx.size();
    }
    out.f_off.reserve(nf); out.f_m.reserve(nf); out.f_k.reserve(nf); out.f_rows.reserve(nf);
    out.f_xoff.reserve(nf); out.f_p0.reserve(nf); out.f_uoff.reserve(nf); out.f_woff.reserve(nf);
    out.f_parent.reserve(nf); out.f_level.reserve(nf); out.f_relmap.reserve(nf); out.f_asm.reserve(nf + 1);
    out.f_child_ptr.reserve(nf + 1); out.f_children.reserve(nf);
    out.rows.reserve(nr); out.relmap.reserve(nr);
    out.asm_tgt.reserve(ne); out.asm_sp.reserve(ne + 1); out.asm_src.reserve(nsrc);
    out.gidx.reserve(nx);
  }
  for (int s = 0; s < nsd; s++) {
    merge(pieces[(size_t)s], out);
    MfBatch().rows.swap(pieces[(size_t)s].rows);  // release as we go
  }
  finalize(out);
}

void mf_build_single(const Csr &M, const MfOptions &opt, MfBatch &out) {
  out = MfBatch();
  int n = M.nrows;
  Work w;
  std::vector<int> &lr = w.lr, &lc = w.lc, &gid = w.gid;
  std::vector<int64_t> &src = w.src;
  gid.resize((size_t)n);
  for (int i = 0; i < n; i++) {
    gid[(size_t)i] = i;
    for (int64_t e = M.ptr[(size_t)i]; e < M.ptr[(size_t)i + 1]; e++) {
      lr.push_back(i); lc.push_back(M.col[(size_t)e]); src.push_back(e);
    }
  }
  dissect(w, n, opt.leaf);
  std::vector<LevelSums> sums;
  add_sums(w.L, sums);
  join(w, plan_joins(sums, opt));
  place_entries(w);
  append(w.L, gid, out);
  finalize(out);
}

}  // namespace dg
