// Compiler and checking interpreter of the dot-product programs.
#include "gox_dot.hpp"
#include "gox_sums.hpp"

#include <algorithm>
#include <cmath>
#include <numeric>
#include <queue>
#include <stdexcept>

namespace gox {

namespace {

// Rough cycles of n products on one warp (only their proportions matter:
// they balance bins and warps)
double sum_cost(int n) { return 60.0 + 25.0 * n; }

struct Writer {
  std::vector<uint32_t> w;
  size_t last = (size_t)-1;  // word index of the header a barrier can go with
  int idle = 0;              // barriers to take without work
  void raw(uint32_t x, uint32_t y, uint32_t z, uint32_t v) { w.insert(w.end(), {x, y, z, v}); }
  // room for n quads in the chunk (and for the quad that leaves it)
  void room(int n) {
    const int used = (int)(w.size() / 4) % kDotChunk;
    if (used + n + 1 <= kDotChunk) return;
    raw(DOT_SKIP, 0u, 0u, 0u);
    while (w.size() % (4 * kDotChunk)) w.push_back(0);
  }
  void flush() {
    if (!idle) return;
    room(1);
    raw(DOT_BAR, (uint32_t)idle, 0u, 0u);
    idle = 0;
  }
  // a sum's products [0, n) as units of up to 8
  void sum(uint32_t op, uint32_t y, uint32_t z, const int32_t* a, const int32_t* b, int n) {
    flush();
    bool cin = false;
    do {
      const int m = std::min(n, kDotTerms);
      room(1 + (m + 1) / 2);
      last = w.size();
      raw(op | (op == DOT_U && !cin && m == n ? DOT_PLAIN : 0u) | (cin ? DOT_CIN : 0u) | (m < n ? DOT_COUT : 0u) |
              ((uint32_t)m << 12), y, z, 0u);
      for (int t = 0; t < m; t += 2) {
        const int u = t + 1 < m ? t + 1 : t;
        raw((uint32_t)a[t], (uint32_t)b[t], (uint32_t)a[u], (uint32_t)b[u]);
      }
      a += m;
      b += m;
      n -= m;
      cin = true;
    } while (n > 0);
  }
  // four sums of m products each (the last ones repeated to make four: the
  // same sum twice stores the same value twice)
  struct Sum { int32_t v, t0; };
  void pack(const Sums& S, const Sum* x, int cnt, int m, bool row, bool first, int ns) {
    flush();
    room(2 + 2 * m);
    last = w.size();
    raw(DOT_PACK | (row ? DOT_ROW : 0u) | (first ? DOT_FIRST : 0u) | ((uint32_t)m << 12), 0u, 0u, 0u);
    auto at = [&](int i) { return x[std::min(i, cnt - 1)]; };
    auto val = [&](int i) { return (uint32_t)(row ? at(i).v - ns : at(i).v); };
    raw(val(0), val(1), val(2), val(3));
    for (int t = 0; t < m; t++) {
      auto a = [&](int i) { return (uint32_t)S.a[at(i).t0 + t]; };
      auto b = [&](int i) { return (uint32_t)S.b[at(i).t0 + t]; };
      raw(a(0), a(1), a(2), a(3));
      raw(b(0), b(1), b(2), b(3));
    }
  }
  // backward rows in a row, in one chunk each
  void chain(const Schedule& sc, const std::vector<int32_t>& rows) {
    flush();
    for (size_t i = 0; i < rows.size();) {
      size_t e = i;
      int q = 1;
      auto quads = [&](int k) { return 1 + (sc.bw_ptr[k + 1] - sc.bw_ptr[k] + 1) / 2; };
      while (e < rows.size() && q + quads(rows[e]) < kDotChunk) q += quads(rows[e++]);
      // (a chunk has room for 5 rows at least; what is left of one is used when
      // it holds a row or two more)
      const int left = kDotChunk - 1 - (int)(w.size() / 4) % kDotChunk;
      if (q > left) {
        size_t f = i;
        int z = 1;
        while (f < rows.size() && z + quads(rows[f]) <= left) z += quads(rows[f++]);
        if (f >= i + 2) {
          e = f;
          q = z;
        }
      }
      room(q);
      last = w.size();
      raw(DOT_CHAIN, (uint32_t)(e - i), 0u, 0u);
      for (size_t r = i; r < e; r++) {
        const int k = rows[r], t0 = sc.bw_ptr[k], n = sc.bw_ptr[k + 1] - t0;
        const bool next = r > i && n > 0 && sc.bw_col[t0] == rows[r - 1];
        raw((uint32_t)k, (uint32_t)sc.diag_slot[k], (uint32_t)n | (next ? DOT_NEXT : 0u), 0u);
        for (int t = 0; t < n; t += 2) {
          const int u = t + 1 < n ? t + 1 : t;
          raw((uint32_t)sc.bw_slot[t0 + t], (uint32_t)sc.bw_col[t0 + t], (uint32_t)sc.bw_slot[t0 + u],
              (uint32_t)sc.bw_col[t0 + u]);
        }
      }
      i = e;
    }
  }
  void fin(int diag, int ll) {
    flush();
    room(1);
    last = w.size();
    raw(DOT_FIN, (uint32_t)diag, (uint32_t)ll, 0u);
  }
  // LU slots and rows, up to 40 of each
  void touch(const std::vector<int32_t>& lu, const std::vector<int32_t>& x) {
    if (lu.empty() && x.empty()) return;
    flush();
    const int ql = ((int)lu.size() + 3) / 4, qx = ((int)x.size() + 3) / 4;
    room(1 + ql + qx);
    raw(DOT_TOUCH, (uint32_t)ql, (uint32_t)qx, 0u);
    for (const std::vector<int32_t>* l : {&lu, &x})
      for (size_t i = 0; i < l->size(); i += 4) {
        auto at = [&](size_t q) { return (uint32_t)(*l)[std::min(q, l->size() - 1)]; };
        raw(at(i), at(i + 1), at(i + 2), at(i + 3));
      }
  }
  void bar() {
    if (idle == 0 && last != (size_t)-1) w[last] |= DOT_BARF;
    else idle++;
    last = (size_t)-1;
  }
  void end() {
    flush();
    room(1);
    raw(DOT_END, 0u, 0u, 0u);
    while (w.size() % (4 * kDotChunk)) w.push_back(0);
    w.insert(w.end(), 4 * kDotChunk * kDotAhead, 0u);
  }
};

void append(DotProgram& P, std::vector<int32_t>& starts, Writer& W) {
  W.end();
  starts.push_back((int32_t)(P.words.size() / 4));
  P.words.insert(P.words.end(), W.w.begin(), W.w.end());
}

}  // namespace

// 16 warps in FP64: more of them only queue for the FP64 pipe (2 lanes a
// cycle), and 32 leave too few registers for 8 products in flight.
static int top_warps(int elem) { return elem == 4 ? 32 : 16; }

// Bins: the more there are, the more of the chip the bottom fills but the more
// columns are left to the ticks (measured, ms per refactor with 32 / 64 / 128 /
// 256 / 512 / 1024 / 2048 bins and no mid stage: 2,000 buses, 128 groups FP32 - / 1.93
// / 1.79 / 1.77 / 1.78 / - / -; 10,000 buses, 128 groups - / 7.4 / 6.4 / 6.1 / 6.0 /
// - / -; with a mid stage: 2,000 buses, one group - / - / .84 / .78 / .73 / - / -;
// 20,000 buses, one group - / - / - / 2.63 / 1.96 / 1.75 / 1.67).  Below 400 unknowns
// the launches around the top cost what the bottom saves (118 buses FP64, one
// group: no bins 0.221, 32 bins 0.219).
// Mid stage: while its CTAs of all groups find an SM each, it takes the early,
// wide ticks off the one SM of a group (ms per refactor without and with 4 / 8 /
// 16 / 32 CTAs: 2,000 buses, one group FP32, 256 bins .99, .79 / .78 / .81 / .83;
// 32 groups 1.03, .84 / .86 / - / -; 128 groups 1.46, - / 1.59; 47 groups FP64
// 2.07, 1.74 with 3 and 1.95 with 8; 20,000 buses, one group 3.86, 2.32 / 2.00 /
// 1.96 / -; 118 buses, one group FP64 .196, .156 with 8).
constexpr int kSMs = 152;

bool dot_few(const DotPlan& p, int groups) { return groups * std::max(p.mid, 3) <= kSMs; }

DotPlan dot_default(const Schedule& sc, int elem, int groups) {
  DotPlan p;
  p.top_warps = top_warps(elem);
  p.chain = dot_chain_terms(elem);
  const bool few = groups * 3 <= kSMs;
  const int per = few ? 8 : 32;  // unknowns per bin
  while (sc.n_u >= 400 && p.bins < (few ? 2048 : 512) && p.bins * per < sc.n_u) p.bins = p.bins ? 2 * p.bins : 32;
  if (few && sc.n_u >= 100) p.mid = std::min(kSMs / groups, sc.n_u >= 20000 ? 16 : 8);
  return p;
}

std::vector<DotPlan> dot_candidates(const Schedule& sc, int elem, int groups) {
  std::vector<DotPlan> out;
  for (int bins : {0, 32, 64, 128, 256, 512, 1024, 2048}) {
    if (bins > 0 && (bins * 4 > sc.n_u || bins * 400 < sc.n_u)) continue;
    if (bins == 0 && sc.n_u > 1500) continue;
    for (int mid : {0, 3, 4, 8, 16, 32}) {
      if (mid > 0 && (mid * groups > kSMs || mid * 20 > sc.n_u || (bins > 0 && bins * 64 < sc.n_u))) continue;
      for (int w : {32, 16}) {
        if (w > top_warps(elem) || (mid > 0 && w < top_warps(elem))) continue;
        DotPlan p;
        p.bins = bins;
        p.mid = mid;
        p.top_warps = w;
        p.chain = dot_chain_terms(elem);
        out.push_back(p);
      }
    }
  }
  return out;
}

void build_dot(const Schedule& sc, const DotPlan& plan, DotProgram& P) {
  if (!dot_fits(sc)) throw std::runtime_error("too many slots for a dot program");
  P = DotProgram();
  P.plan = plan;
  const int n = sc.n_u, ns = sc.n_slots;
  const bool subst = sc.fuse_fwd;
  P.with_subst = subst;
  const Sums S = make_sums(sc);
  auto nt = [&](int v) { return S.ptr[v + 1] - S.ptr[v]; };
  auto len = [&](int k) { return sc.c_ulen[k] + 1 + sc.c_llen[k]; };
  std::vector<int32_t> taken(ns + n, 0);  // products already in the program, per value

  // ---- bottom: parts of the elimination forest of at most cap * (total /
  // bins) cost, grown column by column (a column joins when everything it
  // depends on is in the bottom and the part it makes stays small enough)
  Parts parts(sc, S);
  const std::vector<char>& stage = parts.stage;
  std::vector<int32_t> cta(n, -1);  // the mid column's CTA
  std::vector<std::vector<int32_t>> bin, mid;
  if (plan.bins > 0) {
    parts.grow(0, plan.cap * parts.cost_from(0) / plan.bins);
    bin = parts.deal(0, plan.bins);
  }
  if (plan.mid > 0) {
    parts.grow(1, plan.mid_cap * parts.cost_from(1) / plan.mid);
    for (auto& m : parts.deal(1, plan.mid)) {
      if (m.empty()) continue;
      std::sort(m.begin(), m.end());
      for (int k : m) cta[k] = (int)mid.size();
      mid.push_back(std::move(m));
    }
  }
  const int bottom_cols = (int)std::count(stage.begin(), stage.end(), 0);
  auto emit_sum = [&](Writer& W, uint32_t op, int v, uint32_t z, int t0, int t1) {
    const bool y = v >= ns;
    W.sum(op | (y && t0 == S.ptr[v] ? DOT_FIRST : 0u), (uint32_t)(y ? v - ns : v), z, S.a.data() + t0,
          S.b.data() + t0, t1 - t0);
  };
  // independent sums of one warp (products [t0, t1) of value v): the short ones
  // by fours, those of one length together, the long ones one by one
  struct Part { int32_t v, t0, t1; };
  auto emit_group = [&](Writer& W, const std::vector<Part>& g) {
    std::vector<Writer::Sum> by[3][4];  // LU, y, y from its start; by length
    for (const Part& x : g) {
      const int m = x.t1 - x.t0, kind = x.v < ns ? 0 : x.t0 == S.ptr[x.v] ? 2 : 1;
      if (m == 0 && kind < 2) continue;
      if (m > plan.pack) emit_sum(W, x.v >= ns ? DOT_Y : DOT_U, x.v, 0, x.t0, x.t1);
      else by[kind][m].push_back({x.v, x.t0});
    }
    for (int kind = 0; kind < 3; kind++)
      for (int m = 0; m < 4; m++) {
        const auto& l = by[kind][m];
        for (size_t i = 0; i < l.size(); i += 4) {
          const int cnt = (int)std::min<size_t>(4, l.size() - i);
          if (cnt == 1) emit_sum(W, kind ? DOT_Y : DOT_U, l[i].v, 0, l[i].t0, l[i].t0 + m);
          else W.pack(S, &l[i], cnt, m, kind > 0, kind == 2, ns);
        }
      }
  };
  // a bin's sums by their depth in it (a column's L entries are final one
  // deeper than its deepest sum): those of one depth are independent
  {
    std::vector<int32_t> depth(ns + n, 0);
    std::vector<std::vector<Part>> at;
    std::vector<std::vector<int32_t>> fins;
    for (int b = 0; b < plan.bins; b++) {
      if (bin[b].empty()) continue;
      at.clear();
      fins.clear();
      auto grow = [&](int d) {
        if ((int)at.size() <= d) {
          at.resize(d + 1);
          fins.resize(d + 1);
        }
      };
      auto sum_depth = [&](int v) {
        int d = 0;
        for (int e = S.ptr[v]; e < S.ptr[v + 1]; e++)
          d = std::max({d, depth[S.a[e]], depth[v >= ns ? ns + S.b[e] : S.b[e]]});
        grow(d);
        at[d].push_back({v, S.ptr[v], S.ptr[v + 1]});
        taken[v] = nt(v);
        return d + 1;  // what reads it comes after
      };
      for (int k : bin[b]) {
        const int base = sc.c_base[k], ul = sc.c_ulen[k];
        int f = 0;
        for (int v = base; v < base + len(k); v++) {
          depth[v] = nt(v) ? sum_depth(v) : 0;
          if (v >= base + ul) f = std::max(f, depth[v]);
        }
        grow(f);
        fins[f].push_back(k);
        for (int v = base + ul; v < base + len(k); v++) depth[v] = f + 1;
        if (subst) depth[ns + k] = sum_depth(ns + k);
      }
      Writer W;
      for (size_t d = 0; d < at.size(); d++) {
        emit_group(W, at[d]);
        for (int k : fins[d]) W.fin(sc.diag_slot[k], sc.c_llen[k]);
      }
      append(P, P.bottom, W);
    }
  }
  // ---- prep: per later column, the leading products of each sum whose values
  // the bottom (or the prep of this same column) finishes
  if (bottom_cols > 0) {
    std::vector<int32_t> prep_depth(ns + n, 0);
    std::vector<std::vector<Part>> at;  // the stream's sums, by depth among its columns' U entries
    int left_cols = n - bottom_cols, in_stream = 0;
    // (two columns fill the packs better; four leave too few warps in flight:
    // 2,000 buses, 256 bins, 128 groups FP32 0.305 / 0.276 / 0.285 ms for 1 / 2 / 4)
    const int per_stream = left_cols >= 256 ? 2 : 1;
    for (int k = 0; k < n; k++) {
      if (stage[k] == 0) continue;
      const int base = sc.c_base[k];
      auto prefix = [&](int v) {
        int t = S.ptr[v], d = 0;
        for (; t < S.ptr[v + 1]; t++) {
          if (stage[S.col[S.a[t]]] > 0) break;  // an L value of a later column
          if (v >= ns ? stage[S.b[t]] > 0 : taken[S.b[t]] != nt(S.b[t])) break;
          if (v < ns) d = std::max(d, prep_depth[S.b[t]]);
        }
        if (t == S.ptr[v]) return;
        if ((int)at.size() <= d) at.resize(d + 1);
        at[d].push_back({v, S.ptr[v], t});
        prep_depth[v] = d + 1;
        taken[v] = t - S.ptr[v];
      };
      for (int d = 0; d < len(k); d++) prefix(base + d);
      if (subst) prefix(ns + k);
      left_cols--;
      if ((++in_stream < per_stream && left_cols > 0) || at.empty()) continue;
      Writer W;
      for (auto& g : at) emit_group(W, g);
      append(P, P.prep, W);
      at.clear();
      in_stream = 0;
    }
  }

  // ---- top and mid: nodes (a leading part of a sum, a U entry, a column's pivot
  // and L entries, a y), each in a tick after the ticks of what it reads
  struct Node {
    int32_t kind;    // 0 part, 1 U, 2 column, 3 y
    int32_t v;       // value, or the column
    int32_t t0, t1;  // products (kinds 0, 1, 3)
    int32_t tick;    // as soon as possible
    int32_t late;    // as late as possible
    double cost;
  };
  std::vector<Node> nodes;
  std::vector<std::pair<int32_t, int32_t>> edges;
  std::vector<int32_t> node_of(ns + n, -1);  // value -> the node that finishes it (-1: before the top)
  std::vector<int32_t> done(ns + n, -1);     // value -> tick it is final after
  std::vector<int32_t> from(ns + n, 0);      // first product left for the node that finishes it
  std::vector<int32_t> stop(S.ptr.begin() + 1, S.ptr.end());  // and the end of the products run here
  const int NT = plan.top_warps;
  int makespan = 0;
  std::vector<int32_t> preds;
  // what each tick's warps do
  struct Do { int32_t w; uint32_t op; int32_t v; uint32_t z; int32_t t0, t1; };
  struct Ticks {
    std::vector<std::vector<Do>> plan;
    std::vector<std::vector<double>> load;
  };
  auto add_node = [&](Node nd) {
    std::sort(preds.begin(), preds.end());
    preds.erase(std::unique(preds.begin(), preds.end()), preds.end());
    const int id = (int)nodes.size();
    for (int p : preds)
      if (p >= 0) edges.push_back({p, id});
    nodes.push_back(nd);
    makespan = std::max(makespan, nd.tick + 1);
    return id;
  };
  auto second = [&](int v, int t) { return v >= ns ? ns + S.b[t] : S.b[t]; };
  auto ready = [&](int v, int t0, int t1) {
    int r = -1;
    for (int t = t0; t < t1; t++) r = std::max({r, done[S.a[t]], done[second(v, t)]});
    return r + 1;
  };
  auto take_preds = [&](int v, int t0, int t1) {
    for (int t = t0; t < t1; t++) {
      preds.push_back(node_of[S.a[t]]);
      preds.push_back(node_of[second(v, t)]);
    }
  };
  // a long sum whose last products come late: its leading ones run as parts in
  // earlier ticks, so the tick that finishes it has few left
  constexpr int kPartMin = 3, kPartMax = 8;
  auto split = [&](int v, int final_tick) {
    int t = S.ptr[v] + taken[v];
    const int t1 = stop[v];
    int prev = -1, prev_tick = -1;
    while (t1 - t >= kPartMin) {
      int q = t, r = std::max(0, prev_tick + 1);
      while (q < t1 && q - t < kPartMax) {
        const int rq = std::max(r, ready(v, q, q + 1));
        if (rq > final_tick - 1) break;
        r = rq;
        q++;
      }
      if (q - t < kPartMin) break;
      preds.clear();
      take_preds(v, t, q);
      preds.push_back(prev);
      prev = add_node({0, v, t, q, r, 0, sum_cost(q - t)});
      prev_tick = r;
      t = q;
    }
    from[v] = t;
    return prev;
  };
  auto left = [&](int v) { return stop[v] - from[v]; };
  // the ticks of a CTA's columns (part: of their sums' products up to `stop`)
  auto schedule = [&](const std::vector<int32_t>& columns, bool part) {
    nodes.clear();
    edges.clear();
    makespan = 0;
    for (int k : columns) {
      const int base = sc.c_base[k], ul = sc.c_ulen[k];
      auto sum = [&](int kind, int v) {
        const int r = ready(v, S.ptr[v] + taken[v], stop[v]);
        const int p = split(v, r);
        preds.clear();
        take_preds(v, from[v], stop[v]);
        preds.push_back(p);
        node_of[v] = add_node({kind, v, from[v], stop[v], r, 0, sum_cost(left(v))});
        done[v] = r;
      };
      for (int v = base; v < base + (part ? len(k) : ul); v++)
        if (stop[v] > S.ptr[v] + taken[v]) sum(1, v);
      if (part) {
        if (subst && stop[ns + k] > S.ptr[ns + k] + taken[ns + k]) sum(3, ns + k);
        continue;
      }
      int r = 0;
      for (int v = base + ul; v < base + len(k); v++) r = std::max(r, ready(v, S.ptr[v] + taken[v], S.ptr[v + 1]));
      std::vector<int32_t> cp;
      double cost = 0;
      for (int v = base + ul; v < base + len(k); v++) {
        cp.push_back(split(v, r));
        cost += sum_cost(left(v));
      }
      preds = cp;
      for (int v = base + ul; v < base + len(k); v++) take_preds(v, from[v], S.ptr[v + 1]);
      const int id = add_node({2, k, 0, 0, r, 0, cost});
      for (int v = base + ul; v < base + len(k); v++) {
        node_of[v] = id;
        done[v] = r;
      }
      if (subst && (taken[ns + k] < nt(ns + k) || taken[ns + k] == 0)) sum(3, ns + k);
    }
    // as late as possible
    const int nn = (int)nodes.size();
    for (auto& x : nodes) x.late = makespan - 1;
    std::vector<int32_t> sptr(nn + 1, 0), succ(edges.size()), npred(nn, 0);
    for (auto& e : edges) {
      sptr[e.first + 1]++;
      npred[e.second]++;
    }
    for (int i = 0; i < nn; i++) sptr[i + 1] += sptr[i];
    {
      std::vector<int32_t> at(sptr.begin(), sptr.end() - 1);
      for (auto& e : edges) succ[at[e.first]++] = e.second;
    }
    for (int i = nn - 1; i >= 0; i--)
      for (int q = sptr[i]; q < sptr[i + 1]; q++) nodes[i].late = std::min(nodes[i].late, nodes[succ[q]].late - 1);

    Ticks out;
    std::vector<std::vector<Do>>& plan_of = out.plan;
    std::vector<std::vector<double>>& load_of = out.load;
    int tick = 0;
    auto emit = [&](int w, uint32_t op, int v, uint32_t z, int t0, int t1) {
      plan_of.back().push_back({w, op, v, z, t0, t1});
    };

    // ticks: what cannot wait, then ready nodes (the most urgent first) while
    // the warps have room beside it
    {
      using Item = std::pair<int32_t, int32_t>;  // late, node
      std::priority_queue<Item, std::vector<Item>, std::greater<>> q;
      for (int i = 0; i < nn; i++)
        if (npred[i] == 0) q.push({nodes[i].late, i});
      int todo = nn;
      std::vector<int32_t> now;
      std::vector<double> load(NT);
      while (todo > 0) {
        now.clear();
        double room = 0, sum = 0, ready_cost = 0;
        std::vector<Item> rest;
        while (!q.empty()) {
          Item it = q.top();
          q.pop();
          ready_cost += nodes[it.second].cost;
          if (it.first <= tick) {
            now.push_back(it.second);
            sum += nodes[it.second].cost;
            room = std::max(room, nodes[it.second].kind == 2 ? 250.0 : nodes[it.second].cost);
          } else {
            rest.push_back(it);
          }
        }
        room = std::max({room, 250.0, std::min(ready_cost / NT, 6000.0)});
        for (Item& it : rest) {
          if (sum + nodes[it.second].cost <= 0.8 * room * NT) {
            now.push_back(it.second);
            sum += nodes[it.second].cost;
          } else {
            q.push(it);
          }
        }
        // warps: columns first (split over warps while there are warps for all
        // their entries), then the other sums onto the least loaded warp
        std::fill(load.begin(), load.end(), 0.0);
        plan_of.emplace_back();
        std::vector<int32_t> cols, others, whole;
        for (int i : now) (nodes[i].kind == 2 ? cols : others).push_back(i);
        std::stable_sort(cols.begin(), cols.end(), [&](int x, int y) { return nodes[x].late < nodes[y].late; });
        int used = 0, mids = 0;
        const int shift = (tick * 7) % NT;
        auto least = [&]() { return (int)(std::min_element(load.begin(), load.end()) - load.begin()); };
        for (int i : cols) {
          const int k = nodes[i].v, ul = sc.c_ulen[k], ll = sc.c_llen[k], base = sc.c_base[k];
          if (ll > 0 && used + 1 + ll <= NT && mids < kDotMaxMid) {
            const uint32_t z = (uint32_t)(32 * (1 + ll)) | ((uint32_t)mids << 16), id = (uint32_t)(mids + 1) << 8;
            mids++;
            for (int e = 0; e <= ll; e++) {
              const int v = base + ul + e, w = (used++ + shift) % NT;
              emit(w, (e ? DOT_LH : DOT_D) | id, v, z, from[v], S.ptr[v + 1]);
              load[w] += sum_cost(left(v)) + (e ? 60 : 0);
            }
          } else {
            whole.push_back(i);
          }
        }
        for (int i : whole) {
          const int k = nodes[i].v, ul = sc.c_ulen[k], ll = sc.c_llen[k], base = sc.c_base[k];
          const int w = least();
          for (int e = 0; e <= ll; e++) {
            const int v = base + ul + e;
            if (left(v)) emit(w, DOT_U, v, 0, from[v], S.ptr[v + 1]);
            load[w] += sum_cost(left(v));
          }
          plan_of.back().push_back({w, DOT_FIN, k, 0u, 0, 0});
        }
        std::stable_sort(others.begin(), others.end(), [&](int x, int y) { return nodes[x].cost > nodes[y].cost; });
        for (int i : others) {
          const Node& nd = nodes[i];
          const int w = least();
          const bool y = nd.v >= ns;
          emit(w, y ? DOT_Y : DOT_U, nd.v, 0, nd.t0, nd.t1);
          load[w] += nd.cost;
        }
        load_of.push_back(load);
        todo -= (int)now.size();
        tick++;
        for (int i : now)
          for (int s = sptr[i]; s < sptr[i + 1]; s++)
            if (--npred[succ[s]] == 0) q.push({nodes[succ[s]].late, succ[s]});
      }
    }
    for (int k : columns) {  // (for a later launch all of this is done before)
      auto ran = [&](int v) {
        node_of[v] = done[v] = -1;
        taken[v] = stop[v] - S.ptr[v];
        stop[v] = S.ptr[v + 1];
      };
      for (int v = sc.c_base[k]; v < sc.c_base[k] + len(k); v++) ran(v);
      if (subst) ran(ns + k);
    }
    return out;
  };
  auto row = [&](Writer& w, int k) {
    w.sum(DOT_B, (uint32_t)k, (uint32_t)sc.diag_slot[k], sc.bw_slot.data() + sc.bw_ptr[k],
          sc.bw_col.data() + sc.bw_ptr[k], sc.bw_ptr[k + 1] - sc.bw_ptr[k]);
  };
  // ---- a CTA's backward rows, level by level
  std::vector<int32_t> lev(n, 0);
  auto backward = [&](const std::vector<int32_t>& columns) {
    Ticks out;
    std::vector<std::vector<Do>>& back_of = out.plan;
    std::vector<std::vector<double>>& back_load = out.load;
    std::vector<std::vector<int32_t>> bylev;
    for (size_t i = columns.size(); i-- > 0;) {
      const int k = columns[i];
      int l = 0;
      for (int t = sc.bw_ptr[k]; t < sc.bw_ptr[k + 1]; t++) {
        const int j = sc.bw_col[t];
        if (stage[j] > stage[k]) continue;  // an earlier launch's
        if (stage[j] < stage[k] || cta[j] != cta[k]) throw std::runtime_error("a row reads a later launch's");
        l = std::max(l, lev[j] + 1);
      }
      lev[k] = l;
      if ((int)bylev.size() <= l) bylev.resize(l + 1);
      bylev[l].push_back(k);
    }
    // levels of a row or two, one after the other, are one warp's chain and one
    // tick's: what a row reads of the one before is in a register (its first
    // product), of those before that the warp's own, and no barrier lies
    // between them
    constexpr int kChainRows = 16;
    std::vector<std::vector<int32_t>> ticks_of;
    std::vector<char> chained;
    auto fits = [&](int prev, int k) {
      const int t0 = sc.bw_ptr[k], m = sc.bw_ptr[k + 1] - t0;
      if (m > plan.chain) return false;
      for (int t = 1; t < m; t++)
        if (sc.bw_col[t0 + t] == prev) return false;
      return true;
    };
    for (auto& rows : bylev) {
      bool ok = rows.size() <= 2;
      int prev = !chained.empty() && chained.back() ? ticks_of.back().back() : -1;
      for (int k : rows) {
        ok = ok && fits(prev, k);
        prev = k;
      }
      if (ok && !chained.empty() && chained.back() && ticks_of.back().size() + rows.size() <= (size_t)kChainRows) {
        ticks_of.back().insert(ticks_of.back().end(), rows.begin(), rows.end());
      } else {
        chained.push_back(ok);
        ticks_of.push_back(rows);
      }
    }
    int turn = 0;
    for (size_t t = 0; t < ticks_of.size(); t++) {
      const std::vector<int32_t>& rows = ticks_of[t];
      if (chained[t]) {
        std::vector<double> load(kDotBackWarps, 0.0);
        back_of.emplace_back();
        const int w = turn++ % kDotBackWarps;
        for (int k : rows) back_of.back().push_back({w, DOT_CHAIN, ns + k, 0u, 0, 0});
        load[w] = 1e6;
        back_load.push_back(load);
        continue;
      }
      std::vector<double> load(kDotBackWarps, 0.0);
      back_of.emplace_back();
      for (int k : rows) {
        const int w = rows.size() <= (size_t)kDotBackWarps ? turn++ % kDotBackWarps
                                                : (int)(std::min_element(load.begin(), load.end()) - load.begin());
        load[w] += sum_cost(sc.bw_ptr[k + 1] - sc.bw_ptr[k]);
        back_of.back().push_back({w, DOT_B, ns + k, 0u, 0, 0});
      }
      back_load.push_back(load);
    }
    return out;
  };
  // a CTA's streams; a value whose last use lies too far back to be still in
  // the L1 is touched `ahead` ticks before the tick that needs it, by the
  // warps with the least to do there (not for ticks that fill all warps: they
  // hide their loads behind each other)
  auto streams = [&](Ticks&& ticks, int NT, std::vector<int32_t>& out) {
    const std::vector<std::vector<Do>>& plan_of = ticks.plan;
    std::vector<std::vector<double>>& load_of = ticks.load;
    const int nticks = (int)plan_of.size();
    std::vector<std::vector<std::pair<std::vector<int32_t>, std::vector<int32_t>>>> touch(nticks);  // per tick and warp
    if (plan.ahead > 0) {
      std::vector<int64_t> last(ns + n, -(int64_t)1 << 40);
      int64_t now = 0;
      std::vector<int32_t> need;
      for (int t = 0; t < nticks; t++) {
        need.clear();
        auto use = [&](int v) {
          if (now - last[v] > plan.keep) need.push_back(v);
          last[v] = now++;
        };
        for (const Do& d : plan_of[t]) {
          if (d.op == DOT_FIN) {
            for (int v = sc.diag_slot[d.v]; v <= sc.diag_slot[d.v] + sc.c_llen[d.v]; v++) use(v);
            continue;
          }
          use(d.v);
          if (d.op == DOT_B || d.op == DOT_CHAIN) {
            const int k = d.v - ns;
            use(sc.diag_slot[k]);
            for (int e = sc.bw_ptr[k]; e < sc.bw_ptr[k + 1]; e++) {
              use(sc.bw_slot[e]);
              use(ns + sc.bw_col[e]);
            }
          } else {
            for (int e = d.t0; e < d.t1; e++) {
              use(S.a[e]);
              use(second(d.v, e));
            }
          }
        }
        const int at = t - plan.ahead;
        if (at < 0 || (int)plan_of[t].size() > 3 * NT || need.empty()) continue;
        if (touch[at].empty()) touch[at].resize(NT);
        std::vector<double>& load = load_of[at];
        for (size_t i = 0; i < need.size(); i += 12) {
          const int w = (int)(std::min_element(load.begin(), load.end()) - load.begin());
          for (size_t q = i; q < std::min(need.size(), i + 12); q++)
            (need[q] >= ns ? touch[at][w].second : touch[at][w].first).push_back(need[q] >= ns ? need[q] - ns : need[q]);
          load[w] += 60.0 + 8.0 * 12;
        }
      }
    }
    std::vector<Writer> W(NT);
    for (int t = 0; t < nticks; t++) {
      // per warp: split columns' entries first, then the independent sums, then
      // the columns they finish
      std::vector<std::vector<Part>> group(NT);
      for (const Do& d : plan_of[t]) {
        if (d.op == DOT_B) row(W[d.w], d.v - ns);
        else if (d.op == DOT_CHAIN) continue;
        else if ((d.op & 15u) == DOT_D || (d.op & 15u) == DOT_LH) emit_sum(W[d.w], d.op, d.v, d.z, d.t0, d.t1);
        else if (d.op != DOT_FIN) group[d.w].push_back({d.v, d.t0, d.t1});
      }
      if (!plan_of[t].empty() && plan_of[t][0].op == DOT_CHAIN) {
        std::vector<int32_t> rows;
        for (const Do& d : plan_of[t]) rows.push_back(d.v - ns);
        W[plan_of[t][0].w].chain(sc, rows);
      }
      for (int w = 0; w < NT; w++) emit_group(W[w], group[w]);
      for (const Do& d : plan_of[t])
        if (d.op == DOT_FIN) W[d.w].fin(sc.diag_slot[d.v], sc.c_llen[d.v]);
      if (!touch[t].empty())
        for (int w = 0; w < NT; w++) {
          auto& x = touch[t][w];
          for (size_t i = 0; i < std::max(x.first.size(), x.second.size()); i += 40) {
            auto cut = [&](const std::vector<int32_t>& l) {
              return std::vector<int32_t>(l.begin() + std::min(i, l.size()), l.begin() + std::min(i + 40, l.size()));
            };
            W[w].touch(cut(x.first), cut(x.second));
          }
        }
      if (t + 1 < nticks)
        for (auto& w : W) w.bar();
    }
    for (auto& w : W) append(P, out, w);
  };
  for (auto& m : mid) streams(schedule(m, false), NT, P.mid);
  std::vector<int32_t> top;
  for (int k = 0; k < n; k++)
    if (stage[k] == 2) top.push_back(k);
  // ---- the top columns' products that the mid stage's values (and the same
  // column's, then final) allow, in ticks too: a column's U entries along a
  // path of the mid stage's columns depend on each other
  if (!mid.empty())
    for (size_t i = 0; i < top.size();) {
      std::vector<int32_t> cols;
      for (; i < top.size() && (int)cols.size() < plan.prep_cols; i++) {
        const int k = top[i], base = sc.c_base[k];
        bool any = false;
        auto prefix = [&](int v) {
          const int t0 = S.ptr[v] + taken[v];
          for (stop[v] = t0; stop[v] < S.ptr[v + 1]; stop[v]++) {
            const int a = S.a[stop[v]], b = S.b[stop[v]];
            if (stage[S.col[a]] > 1 || (v >= ns ? stage[b] > 1 : stop[b] < S.ptr[b + 1])) break;
          }
          any |= stop[v] > t0;
        };
        for (int d = 0; d < len(k); d++) prefix(base + d);
        if (subst) prefix(ns + k);
        if (any) cols.push_back(k);
        else
          for (int d = 0; d < len(k); d++) stop[base + d] = S.ptr[base + d + 1];
        if (!any && subst) stop[ns + k] = S.ptr[ns + k + 1];
      }
      if (!cols.empty()) streams(schedule(cols, true), NT, P.prep2);
    }
  streams(schedule(top, false), NT, P.top);
  if (!subst) return;
  streams(backward(top), kDotBackWarps, P.tback);
  for (auto& m : mid) streams(backward(m), kDotBackWarps, P.midback);
  for (int b = 0; b < plan.bins; b++) {
    if (bin[b].empty()) continue;
    Writer w;
    for (size_t i = bin[b].size(); i-- > 0;) row(w, bin[b][i]);
    append(P, P.back, w);
  }
}

std::string run_dot_host(const Schedule& sc, const DotProgram& P, std::vector<double>& lu,
                         const std::vector<double>& rhs, std::vector<double>& X, bool& singular) {
  const int n = sc.n_u, ns = sc.n_slots;
  const Sums S = make_sums(sc);
  X.assign(n, 0.0);
  singular = false;
  // per value (LU slots, then the solution vector): how many products its sum
  // has taken, whether it is final, who wrote and read it last and when
  std::vector<int32_t> taken(ns + n, 0);
  std::vector<char> fin(ns + n, 0), xdone(n, 0);
  std::vector<int64_t> wtick(ns + n, -1), rtick(ns + n, -1);
  std::vector<int32_t> wwarp(ns + n, -1), rwarp(ns + n, -1);
  // ... and the CTA, of a launch of several CTAs with ticks (numbered through all
  // launches; 0: the launch has none): launch and CTA of the last write and read
  std::vector<int32_t> wlaunch(ns + n, -1), rlaunch(ns + n, -1), wcta(ns + n, -1), rcta(ns + n, -1);
  int32_t launch_no = 0, cta = 0;
  for (int k = 0; k < n; k++)
    for (int v = sc.c_base[k]; v < sc.c_base[k] + sc.c_ulen[k]; v++)
      if (S.ptr[v + 1] == S.ptr[v]) fin[v] = 1;
  if (!P.with_subst)
    for (int k = 0; k < n; k++) fin[ns + k] = 1;
  std::string err;
  const size_t nq = P.words.size() / 4;
  int64_t tick = 0;
  uint32_t may = 0;  // the units the running launch has code for
  auto fail = [&](const char* s) {
    if (err.empty()) err = s;
    return false;
  };
  auto read = [&](int v, int w) {
    if (wtick[v] == tick && wwarp[v] != w) return fail("a value read in the tick another warp writes it");
    if (wlaunch[v] == launch_no && wcta[v] != cta) return fail("a value read in the launch another CTA writes it");
    if (rlaunch[v] != launch_no) { rlaunch[v] = launch_no; rcta[v] = cta; }
    else if (rcta[v] != cta) rcta[v] = -2;
    if (rtick[v] != tick) { rtick[v] = tick; rwarp[v] = w; }
    else if (rwarp[v] != w) rwarp[v] = -2;  // several warps
    return true;
  };
  auto write = [&](int v, int w) {
    if (wtick[v] == tick && wwarp[v] != w) return fail("two warps write one value in one tick");
    if (rtick[v] == tick && rwarp[v] != w) return fail("a value written in the tick another warp reads it");
    if ((wlaunch[v] == launch_no && wcta[v] != cta) || (rlaunch[v] == launch_no && rcta[v] != cta))
      return fail("a value written in the launch another CTA uses it");
    wtick[v] = tick;
    wwarp[v] = w;
    wlaunch[v] = launch_no;
    wcta[v] = cta;
    return true;
  };
  struct Held { uint32_t z, id; };
  struct Warp {
    size_t pos;
    int bars = 0;
    bool ended = false, waits = false;  // waits: at a mid barrier
    double car = 0;
    int carried = -1;                   // value of the open sum
  };
  std::vector<std::pair<uint32_t, double>> mid_inv;  // mid barriers reached by their pivot's warp
  std::vector<Held> held;
  // runs a warp up to its next barrier, a mid barrier nobody reached yet, or its end
  auto step = [&](Warp& A, int w, bool top) -> bool {
    if (!A.waits && A.bars > 0 && --A.bars > 0) return true;
    for (;;) {
      if ((A.pos / kDotChunk + 1 + kDotAhead) * kDotChunk > nq) return fail("a stream runs past the program");
      const uint32_t* h = &P.words[A.pos * 4];
      const uint32_t op = h[0] & 15u;
      if (!((may >> op) & 1u)) return fail("a unit in the wrong launch");
      if (op == DOT_END) {
        A.ended = true;
        return A.carried < 0 || fail("a sum left open");
      }
      if (op == DOT_SKIP) {
        A.pos = (A.pos / kDotChunk + 1) * kDotChunk;
        continue;
      }
      if (op == DOT_BAR) {
        A.pos++;
        A.bars = (int)h[1];
        return (top && A.bars > 0) || fail("a bin with a barrier");
      }
      if (op == DOT_TOUCH) {
        const size_t nt = (size_t)h[1] + h[2];
        if (A.pos % kDotChunk + 1 + nt + 1 > (size_t)kDotChunk || A.pos + 1 + nt > nq) return fail("a unit that leaves its chunk");
        for (size_t i = 0; i < 4 * nt; i++)
          if (h[4 + i] >= (uint32_t)(i < 4 * (size_t)h[1] ? ns : n)) return fail("a touched value out of range");
        A.pos += 1 + nt;
        continue;
      }
      if (op == DOT_PACK) {
        const int m = (int)((h[0] >> 12) & 15u);
        const bool row = (h[0] & DOT_ROW) != 0, first = (h[0] & DOT_FIRST) != 0;
        if (m > 3 || (first && !row)) return fail("a pack out of range");
        if (A.pos % kDotChunk + 2 + 2 * m + 1 > (size_t)kDotChunk || A.pos + 2 + 2 * m > nq)
          return fail("a unit that leaves its chunk");
        if (A.carried >= 0) return fail("a sum left open");
        double out[4];
        for (int i = 0; i < 4; i++) {
          if (h[4 + i] >= (uint32_t)(row ? n : ns)) return fail("a value out of range");
          const int v = row ? ns + (int)h[4 + i] : (int)h[4 + i];
          bool again = false;
          for (int q = 0; q < i; q++)
            if (h[4 + q] == h[4 + i]) {
              again = true;
              for (int t = 0; t < 2 * m; t++)
                if (h[8 + 4 * t + q] != h[8 + 4 * t + i]) return fail("a repeated sum with other products");
            }
          if (again) continue;
          if (fin[v]) return fail("a final value written again");
          if (row && first != (taken[v] == 0)) return fail("a sum that starts twice or not at all");
          if (!first && !read(v, w)) return false;
          double s = first ? rhs[h[4 + i]] : row ? X[h[4 + i]] : lu[v];
          for (int t = 0; t < m; t++) {
            const uint32_t a = h[8 + 8 * t + i], b = h[12 + 8 * t + i];
            if (a >= (uint32_t)ns || b >= (uint32_t)(row ? n : ns)) return fail("a product out of range");
            const int vb = row ? ns + (int)b : (int)b, e = S.ptr[v] + taken[v]++;
            if (!read((int)a, w) || !read(vb, w)) return false;
            if (e >= S.ptr[v + 1] || S.a[e] != (int)a || S.b[e] != (int)b) return fail("a product out of order");
            if (!fin[a] || !fin[vb]) return fail("a product before its value is final");
            s -= lu[a] * (row ? X[b] : lu[b]);
          }
          out[i] = s;
        }
        for (int i = 0; i < 4; i++) {
          const int v = row ? ns + (int)h[4 + i] : (int)h[4 + i];
          bool again = false;
          for (int q = 0; q < i; q++) again |= h[4 + q] == h[4 + i];
          if (again) continue;
          if (!write(v, w)) return false;
          (row ? X[h[4 + i]] : lu[v]) = out[i];
          if ((row || v < sc.diag_slot[S.col[v]]) && taken[v] == S.ptr[v + 1] - S.ptr[v]) fin[v] = 1;
        }
        A.pos += 2 + 2 * m;
      } else if (op == DOT_FIN) {
        const int d = (int)h[1];
        if (h[1] >= (uint32_t)ns || d != sc.diag_slot[S.col[d]] || (int)h[2] != sc.c_llen[S.col[d]])
          return fail("a column out of range");
        for (int v = d; v <= d + (int)h[2]; v++) {
          if (fin[v] || taken[v] != S.ptr[v + 1] - S.ptr[v]) return fail("a column finished before its sums");
          if (!read(v, w) || !write(v, w)) return false;
          fin[v] = 1;
        }
        if (lu[d] == 0) singular = true;
        const double inv = 1.0 / lu[d];
        for (int v = d + 1; v <= d + (int)h[2]; v++) lu[v] = lu[v] * inv;
        A.pos++;
      }
      if (op == DOT_CHAIN) {
        if (A.carried >= 0) return fail("a sum left open");
        size_t q = A.pos + 1;
        int prev = -1;
        for (uint32_t r = 0; r < h[1]; r++) {
          if (q >= nq || q / kDotChunk != A.pos / kDotChunk) return fail("a unit that leaves its chunk");
          const uint32_t* x = &P.words[q * 4];
          const int m = (int)(x[2] & 0xffffu);
          if (x[0] >= (uint32_t)n || m > P.plan.chain) return fail("a chain's row out of range");
          const int k = (int)x[0], v = ns + k;
          if (!fin[v] || !read(v, w)) return fail("x before y is final");
          if (x[1] != (uint32_t)sc.diag_slot[k] || !fin[x[1]] || !read((int)x[1], w))
            return fail("a backward row with another pivot");
          if (m != sc.bw_ptr[k + 1] - sc.bw_ptr[k]) return fail("an incomplete backward row");
          if (q + 1 + (m + 1) / 2 > nq || (q + (m + 1) / 2) / kDotChunk != A.pos / kDotChunk)
            return fail("a unit that leaves its chunk");
          double s = X[k];
          for (int t = 0; t < m; t++) {
            const uint32_t* y = x + 4 + 4 * (t / 2) + 2 * (t & 1);
            const int e = sc.bw_ptr[k] + t;
            if ((uint32_t)sc.bw_slot[e] != y[0] || (uint32_t)sc.bw_col[e] != y[1]) return fail("a backward term out of order");
            if (!fin[y[0]] || !xdone[y[1]]) return fail("a backward term before its x");
            if (!read((int)y[0], w) || !read(ns + (int)y[1], w)) return false;
            // the loads of a row are issued before the row before it is stored
            const bool next = t == 0 && (x[2] & DOT_NEXT);
            if (next != ((int)y[1] == prev)) return fail("a chain's row that misses the one before it");
            s -= lu[y[0]] * X[y[1]];
          }
          const double xx = s / lu[x[1]];
          if (!std::isfinite(xx)) singular = true;
          if (!write(v, w)) return false;
          X[k] = xx;
          xdone[k] = 1;
          prev = k;
          q += 1 + (m + 1) / 2;
        }
        if (q % kDotChunk == 0) return fail("a unit that leaves its chunk");
        A.pos = q;
      }
      if (op == DOT_PACK || op == DOT_FIN || op == DOT_CHAIN) {
        if (h[0] & DOT_BARF) {
          if (!top) return fail("a bin with a barrier");
          A.bars = 1;
          return true;
        }
        continue;
      }
      if ((h[0] & DOT_PLAIN) && (op != DOT_U || (h[0] & (DOT_CIN | DOT_COUT | DOT_FIRST)))) return fail("a plain unit with flags");
      const int m = (int)((h[0] >> 12) & 15u);
      const bool row = op == DOT_Y || op == DOT_B, cin = (h[0] & DOT_CIN) != 0, cout = (h[0] & DOT_COUT) != 0;
      if (op < DOT_U || op > DOT_B || m > kDotTerms || h[1] >= (uint32_t)(row ? n : ns)) return fail("a unit out of range");
      if (A.pos % kDotChunk + 1 + (m + 1) / 2 + 1 > kDotChunk) return fail("a unit that leaves its chunk");
      if (A.pos + 1 + (m + 1) / 2 > nq) return fail("a unit runs past the program");
      const int v = row ? ns + (int)h[1] : (int)h[1];
      double mid = 0;
      if (op == DOT_LH && !cout) {
        const std::pair<uint32_t, double>* x = nullptr;
        for (auto& y : mid_inv)
          if (y.first == ((h[0] >> 8) & 15u)) x = &y;
        A.waits = x == nullptr;
        if (A.waits) return true;
        mid = x->second;
      }
      if (cin != (A.carried >= 0) || (cin && A.carried != v)) return fail("a sum carried to another value");
      A.carried = -1;
      const bool first = op == DOT_Y && (h[0] & DOT_FIRST);
      double s = A.car, d = 0;
      if (!cin) {
        if (!first && !read(v, w)) return false;
        s = first ? rhs[h[1]] : row ? X[h[1]] : lu[v];
      }
      if (op == DOT_B) {
        if (!fin[v]) return fail("x before y is final");
        if (h[2] != (uint32_t)sc.diag_slot[h[1]] || !fin[h[2]]) return fail("a backward row with another pivot");
        if (!read((int)h[2], w)) return false;
        d = lu[h[2]];
        if (!cin) taken[v] = 0;  // counts the backward terms from here on
      } else {
        if (fin[v]) return fail("a final value written again");
        if (op == DOT_Y && !cin && first != (taken[v] == 0)) return fail("a sum that starts twice or not at all");
      }
      for (int t = 0; t < m; t++) {
        const uint32_t* q = h + 4 + 4 * (t / 2) + 2 * (t & 1);
        if (q[0] >= (uint32_t)ns || q[1] >= (uint32_t)(row ? n : ns)) return fail("a product out of range");
        const int b = row ? ns + (int)q[1] : (int)q[1];
        if (!read((int)q[0], w) || !read(b, w)) return false;
        if (op == DOT_B) {
          const int e = sc.bw_ptr[h[1]] + taken[v]++;
          if (e >= sc.bw_ptr[h[1] + 1] || (int)q[0] != sc.bw_slot[e] || (int)q[1] != sc.bw_col[e])
            return fail("a backward term out of order");
          if (!fin[q[0]] || !xdone[q[1]]) return fail("a backward term before its x");
        } else {
          const int e = S.ptr[v] + taken[v]++;
          if (e >= S.ptr[v + 1] || S.a[e] != (int)q[0] || S.b[e] != (int)q[1]) return fail("a product out of order");
          if (!fin[q[0]] || !fin[b]) return fail("a product before its value is final");
        }
        s -= lu[q[0]] * (row ? X[q[1]] : lu[b]);
      }
      A.pos += 1 + (m + 1) / 2;
      if (cout) {
        A.car = s;
        A.carried = v;
        if (h[0] & DOT_BARF) return fail("a barrier inside a sum");
        continue;
      }
      if (!write(v, w)) return false;
      const bool whole = op != DOT_B && taken[v] == S.ptr[v + 1] - S.ptr[v];
      const int k = row ? 0 : S.col[v];
      if (op == DOT_U || op == DOT_Y) {
        (row ? X[h[1]] : lu[v]) = s;
        // a U unit on the pivot or an L entry is a leading part of its sum
        if ((row || v < sc.diag_slot[k]) && whole) fin[v] = 1;
      } else if (op == DOT_D) {
        if (!whole || v != sc.diag_slot[k]) return fail("an incomplete pivot");
        lu[v] = s;
        fin[v] = 1;
        if (s == 0) singular = true;
        const uint32_t id = (h[0] >> 8) & 15u;
        if (id == 0 || !top || id > (uint32_t)kDotMaxMid || (h[2] >> 16) >= (uint32_t)kDotMaxMid)
          return fail("a mid barrier out of range");
        mid_inv.push_back({id, 1.0 / s});
      } else if (op == DOT_LH) {
        if (!whole || v <= sc.diag_slot[k]) return fail("an incomplete L entry");
        if (!fin[sc.diag_slot[k]] || wtick[sc.diag_slot[k]] != tick) return fail("an L entry of another column's pivot");
        held.push_back({h[2], (h[0] >> 8) & 15u});
        lu[v] = s * mid;
        fin[v] = 1;
      } else {
        if (taken[v] != sc.bw_ptr[h[1] + 1] - sc.bw_ptr[h[1]]) return fail("an incomplete backward row");
        const double x = s / d;
        if (!std::isfinite(x)) singular = true;
        X[h[1]] = x;
        xdone[h[1]] = 1;
      }
      if (h[0] & DOT_BARF) {
        if (!top) return fail("a bin with a barrier");
        A.bars = 1;
        return true;
      }
    }
  };
  constexpr uint32_t kAny = 1u << DOT_END | 1u << DOT_SKIP, kTick = kAny | 1u << DOT_BAR | 1u << DOT_TOUCH,
                     kSums = 1u << DOT_PACK | 1u << DOT_FIN | 1u << DOT_U | 1u << DOT_Y;
  auto launch = [&](const std::vector<int32_t>& st, uint32_t units, auto&& run) {
    int w = 0;
    may = units;
    launch_no++;
    cta = 0;
    for (int32_t s : st)
      if (s < 0 || (size_t)s >= nq || !run(s, w++)) return false;
    tick++;
    return true;
  };
  auto bin = [&](int32_t s, int w) {
    Warp B{(size_t)s};
    return step(B, w, false) && (B.ended || fail("a bin that does not end"));
  };
  if (!launch(P.bottom, kAny | kSums, bin) || !launch(P.prep, kAny | kSums, bin)) return err;
  // a CTA's warps, tick by tick
  auto ticks = [&](const std::vector<int32_t>& st, uint32_t units) -> bool {
    may = units;
    const int NT = (int)st.size();
    std::vector<Warp> A;
    for (int32_t s : st) {
      if (s < 0 || (size_t)s >= nq) return fail("a stream out of range");
      A.push_back({(size_t)s});
    }
    for (int ended = 0; ended < NT;) {
      held.clear();
      mid_inv.clear();
      ended = 0;
      // every warp to its barrier; one that waits at a mid barrier goes on when
      // the pivot's warp has arrived there
      std::vector<char> run(NT, 1);
      for (bool moved = true; moved;) {
        moved = false;
        for (int w = 0; w < NT; w++) {
          if (!run[w] || A[w].ended) continue;
          const size_t at = A[w].pos;
          const bool waited = A[w].waits;
          if (!step(A[w], w, true)) return false;
          run[w] = A[w].waits;
          moved |= !A[w].waits || A[w].pos != at || !waited;
        }
      }
      for (int w = 0; w < NT; w++) {
        if (A[w].waits) return fail("a mid barrier that nobody reaches");
        ended += A[w].ended;
      }
      for (auto& m : mid_inv) {
        int cnt = 0;
        for (auto& m2 : mid_inv) cnt += m2.first == m.first;
        uint32_t same = 1;
        for (auto& x : held) same += x.id == m.first;
        if (cnt != 1 || same < 2) return fail("a mid barrier used twice in one tick, or by nobody");
      }
      for (auto& x : held) {
        uint32_t same = 1;
        for (auto& y : held) same += y.id == x.id;
        if ((x.z & 0xffffu) != 32u * same) return fail("a held L entry without its mid barrier");
      }
      if (ended != 0 && ended != NT) return fail("the warps take different numbers of barriers");
      tick++;
    }
    return true;
  };
  // a launch of CTAs of NT warps each
  auto ctas = [&](const std::vector<int32_t>& st, size_t NT, uint32_t units) {
    launch_no++;
    if (st.size() % NT) return fail("a CTA with missing warps");
    for (size_t c = 0; c * NT < st.size(); c++) {
      cta = (int32_t)c;
      if (!ticks(std::vector<int32_t>(st.begin() + c * NT, st.begin() + (c + 1) * NT), units)) return false;
    }
    return true;
  };
  const uint32_t fwd = kTick | kSums | 1u << DOT_D | 1u << DOT_LH, bwd = kTick | 1u << DOT_B | 1u << DOT_CHAIN;
  const size_t NT = (size_t)P.plan.top_warps;
  if (P.top.size() != NT || P.tback.size() > (size_t)kDotBackWarps) return "a top of other than one CTA";
  if (!ctas(P.mid, NT, fwd) || !ctas(P.prep2, NT, fwd) || !ctas(P.top, NT, fwd) ||
      !ctas(P.tback, kDotBackWarps, bwd) || !ctas(P.midback, kDotBackWarps, bwd))
    return err;
  if (!launch(P.back, kAny | 1u << DOT_B, bin)) return err;
  for (int v = 0; v < ns + n; v++)
    if (!fin[v]) return "a value is left unfinished";
  if (P.with_subst)
    for (int k = 0; k < n; k++)
      if (!xdone[k]) return "a row of the solution is left out";
  return err;
}

}  // namespace gox
