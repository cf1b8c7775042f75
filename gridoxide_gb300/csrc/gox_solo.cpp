// Compiler and checking interpreter of the solo programs.
#include "gox_solo.hpp"

#include <algorithm>
#include <cmath>
#include <queue>
#include <stdexcept>

#include "gox_sums.hpp"

namespace gox {

namespace {

// A lane's sum in a tick: products [t0, t1) of value v (backward: of row v's)
struct Lane {
  int32_t v, t0, t1;
  uint32_t info;
};
// 32 lanes that run as many units as their longest sum has
struct Vec {
  std::vector<Lane> lane;
  int units = 1;
  bool col = false;
};
// A CTA's ticks
using Ticks = std::vector<std::vector<Vec>>;

// A schedule that solo programs can be compiled from
bool solo_possible(const Schedule& sc) {
  return sc.fuse_fwd && sc.n_u > 0 && (int64_t)sc.n_slots + sc.n_u < (1 << 28);
}

int units_of(int n) { return std::max(1, (n + kSoloTerms - 1) / kSoloTerms); }

}  // namespace

// The parts' CTAs, ms per refactor of one scenario (three units under way) with 0 / 4 / 8 / 16 / 32 / 64
// (-: its values do not fit): 118 buses FP64 .104 / .126 / .117 / - / - / -, FP32
// .049; 2,000 buses FP32 .540 / .397 / .380 / .367 / .360 / -, FP64 - / .769 /
// .747 / .736 / - / -; 10,000 FP32 - / - / .637 / .592 / .562 / -; 20,000 FP32 - /
// - / - / .905 / .735 / .819.
static bool build_solo(const Schedule& sc, const Sums& S, const SoloPlan& plan, SoloProgram& P);
bool build_solo_default(const Schedule& sc, int elem, bool wide, SoloProgram& out) {
  out = SoloProgram();
  if (!solo_possible(sc)) return false;
  const Sums S = make_sums(sc);
  SoloPlan p;
  p.elem = elem;
  // (the values of the parts together, some twice)
  const double share = 1.2 * elem * ((double)sc.n_slots + sc.n_u) / kSoloMaxBytes;
  const int best = !wide ? 0 : sc.n_u < 1000 ? 0 : sc.n_u < 10000 ? 16 : 32;
  for (int ctas : {0, 4, 8, 16, 32, 64}) {
    if (ctas < best || (ctas > 0 && ctas < share)) continue;
    p.ctas = ctas;
    if (build_solo(sc, S, p, out)) return true;
  }
  return false;
}

int solo_most(const Schedule& sc, int elem) {
  if (!solo_possible(sc)) return 0;
  // one CTA: places by its values; several: an SM has eight places at most, the
  // parts have four CTAs at least
  const int64_t bytes = solo_ring_bytes(kSoloDepth) + ((int64_t)sc.n_slots + sc.n_u + 1) * elem;
  const int64_t one = bytes <= kSoloSmem ? 152 * std::min<int64_t>(8, (228 * 1024) / (bytes + 1024)) : 0;
  return (int)std::max<int64_t>(one, 152 * 8 / 4);
}

int solo_scenarios(const SoloProgram& p, int depth) {
  int most = 1 << 20;
  for (int v : p.max_values)
    if (solo_ring_bytes(depth) + v * p.plan.elem > kSoloSmem) return 0;
  for (int i : {0, 2, 3}) {  // (the second launch's CTAs are many and short)
    const int ctas = (int)p.launch[i].size();
    if (ctas == 0) continue;
    const int bytes = solo_ring_bytes(depth) + p.max_values[i] * p.plan.elem + 1024;
    most = std::min(most, 152 * std::min(8, (228 * 1024) / bytes) / ctas);
  }
  return most;
}

bool build_solo(const Schedule& sc, const SoloPlan& plan, SoloProgram& P) {
  P = SoloProgram();
  return solo_possible(sc) && build_solo(sc, make_sums(sc), plan, P);
}

static bool build_solo(const Schedule& sc, const Sums& S, const SoloPlan& plan, SoloProgram& P) {
  P = SoloProgram();
  P.plan = plan;
  const int max_values = kSoloMaxBytes / plan.elem;
  const int n = sc.n_u, ns = sc.n_slots, zero = ns + n;
  if (plan.ctas == 0 && zero + 1 > max_values) return false;
  auto nt = [&](int v) { return S.ptr[v + 1] - S.ptr[v]; };
  Parts parts(sc, S);
  std::vector<int32_t> cta(n, -1);
  std::vector<std::vector<int32_t>> mid;
  if (plan.ctas > 0) {
    parts.grow(1, parts.cost_from(1) / plan.ctas);
    for (auto& m : parts.deal(1, plan.ctas)) {
      if (m.empty()) continue;
      std::sort(m.begin(), m.end());
      for (int k : m) cta[k] = (int)mid.size();
      mid.push_back(std::move(m));
    }
  }
  const std::vector<char>& stage = parts.stage;
  auto second = [&](int v, int t) { return v >= ns ? ns + S.b[t] : S.b[t]; };
  // The values that the parts' and the rest's CTAs use, before anything is
  // scheduled: a plan they do not fit is left here (20,000 buses FP64, where none
  // fits: 1,480 ms on one core -> 40; 50,000 buses FP32 3,900 -> 95).
  {
    std::vector<int32_t> by(zero, -1), begin(S.ptr.begin(), S.ptr.end() - 1);  // begin: past what the second launch ran
    if (!mid.empty())
      for (int k = 0; k < n; k++) {
        if (stage[k] != 2) continue;
        auto leading = [&](int v) {
          for (int& t = begin[v]; t < S.ptr[v + 1]; t++)
            if (stage[S.col[S.a[t]]] > 1 || (v >= ns ? stage[S.b[t]] > 1 : begin[S.b[t]] < S.ptr[S.b[t] + 1])) break;
        };
        for (int v = sc.c_base[k]; v <= sc.c_base[k] + sc.c_ulen[k] + sc.c_llen[k]; v++) leading(v);
        leading(ns + k);
      }
    int32_t id = 0;
    int64_t used = 0;
    auto use = [&](int v) {
      used += by[v] != id;
      by[v] = id;
    };
    auto sum = [&](int v, bool always) {
      if (always || begin[v] < S.ptr[v + 1]) use(v);
      for (int t = begin[v]; t < S.ptr[v + 1]; t++) {
        use(S.a[t]);
        use(second(v, t));
      }
    };
    auto column = [&](int k) {
      const int d = sc.c_base[k] + sc.c_ulen[k];
      for (int v = sc.c_base[k]; v <= d + sc.c_llen[k]; v++) sum(v, v >= d);
      sum(ns + k, false);
    };
    auto row = [&](int k) {
      use(ns + k);
      use(sc.diag_slot[k]);
      for (int t = sc.bw_ptr[k]; t < sc.bw_ptr[k + 1]; t++) {
        use(sc.bw_slot[t]);
        use(ns + sc.bw_col[t]);
      }
    };
    auto fits = [&]() {
      const bool ok = used + 1 <= max_values;
      id++;
      used = 0;
      return ok;
    };
    for (const auto& m : mid) {
      for (int k : m) column(k);
      if (!fits()) return false;
      for (int k : m) row(k);
      if (!fits()) return false;
    }
    for (int k = 0; k < n; k++)
      if (stage[k] == 2) {
        column(k);
        row(k);
      }
    if (!fits()) return false;
  }
  std::vector<int32_t> taken(ns + n, 0), stop(S.ptr.begin() + 1, S.ptr.end()), done(ns + n, -1), from(ns + n, 0);

  // ---- a CTA's forward ticks: nodes (a leading part of a sum, a sum, a column's
  // pivot and L entries), each in a tick after the ticks of what it reads
  struct Node {
    int32_t v, t0, t1;  // a sum; t1 < 0: column v
    int32_t tick, late, lanes;
  };
  auto forward = [&](const std::vector<int32_t>& columns, bool part) {
    std::vector<Node> nodes;
    std::vector<std::pair<int32_t, int32_t>> edges;
    std::vector<int32_t> preds;
    static thread_local std::vector<int32_t> node_of;
    node_of.assign(ns + n, -1);
    int makespan = 0;
    auto add = [&](Node nd) {
      std::sort(preds.begin(), preds.end());
      preds.erase(std::unique(preds.begin(), preds.end()), preds.end());
      const int id = (int)nodes.size();
      for (int p : preds)
        if (p >= 0) edges.push_back({p, id});
      nodes.push_back(nd);
      makespan = std::max(makespan, nd.tick + 1);
      return id;
    };
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
    // leading products in earlier ticks, a unit each
    auto split = [&](int v, int final_tick) {
      int t = S.ptr[v] + taken[v], prev = -1, prev_tick = -1;
      const int t1 = stop[v];
      while (t1 - t > 0) {
        int q = t, r = std::max(0, prev_tick + 1);
        while (q < t1 && q - t < kSoloTerms) {
          const int rq = std::max(r, ready(v, q, q + 1));
          if (rq > final_tick - 1) break;
          r = rq;
          q++;
        }
        // (one product is worth a unit of its own only where the last tick's
        // would be two)
        if (q == t || (q - t < 2 && t1 - t <= kSoloTerms)) break;
        preds.clear();
        take_preds(v, t, q);
        preds.push_back(prev);
        prev = add({v, t, q, r, 0, 1});
        prev_tick = r;
        t = q;
      }
      from[v] = t;
      return prev;
    };
    auto sum = [&](int v) {
      const int r = ready(v, S.ptr[v] + taken[v], stop[v]);
      const int p = split(v, r);
      preds.clear();
      take_preds(v, from[v], stop[v]);
      preds.push_back(p);
      node_of[v] = add({v, from[v], stop[v], r, 0, 1});
      done[v] = r;
    };
    for (int k : columns) {
      const int base = sc.c_base[k], ul = sc.c_ulen[k], ll = sc.c_llen[k];
      for (int v = base; v < base + (part ? ul + 1 + ll : ul); v++)
        if (stop[v] > S.ptr[v] + taken[v]) sum(v);
      if (stop[ns + k] > S.ptr[ns + k] + taken[ns + k]) sum(ns + k);
      if (part) continue;
      // more L entries than a warp's lanes: the pivot's sum first, in a tick before
      if (ll > 31 && nt(base + ul) > taken[base + ul]) {
        sum(base + ul);
        from[base + ul] = stop[base + ul];
      }
      int r = 0;
      for (int v = base + ul; v < base + ul + 1 + ll; v++) {
        if (v == base + ul && ll > 31) r = std::max(r, done[v] + 1);
        else r = std::max(r, ready(v, S.ptr[v] + taken[v], stop[v]));
      }
      std::vector<int32_t> cp;
      for (int v = base + ul; v < base + ul + 1 + ll; v++) {
        if (v == base + ul && ll > 31) {
          from[v] = stop[v];
          cp.push_back(node_of[v]);
        } else {
          cp.push_back(split(v, r));
        }
      }
      preds = cp;
      for (int v = base + ul; v < base + ul + 1 + ll; v++) take_preds(v, from[v], stop[v]);
      const int id = add({k, 0, -1, r, 0, 1 + ll});
      for (int v = base + ul; v < base + ul + 1 + ll; v++) {
        node_of[v] = id;
        done[v] = r;
      }
    }
    const int nn = (int)nodes.size();
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
    // as late as possible
    for (auto& x : nodes) x.late = makespan - 1;
    for (int i = nn - 1; i >= 0; i--)
      for (int q = sptr[i]; q < sptr[i + 1]; q++) nodes[i].late = std::min(nodes[i].late, nodes[succ[q]].late - 1);
    auto units = [&](const Node& x) {
      if (x.t1 >= 0) return units_of(x.t1 - x.t0);
      int u = 1;
      const int d = sc.c_base[x.v] + sc.c_ulen[x.v];
      for (int v = d; v <= d + sc.c_llen[x.v]; v++) u = std::max(u, units_of(stop[v] - from[v]));
      return u;
    };
    Ticks out;
    using Item = std::pair<int32_t, int32_t>;  // late, node
    std::priority_queue<Item, std::vector<Item>, std::greater<>> q;
    for (int i = 0; i < nn; i++)
      if (npred[i] == 0) q.push({nodes[i].late, i});
    std::vector<int32_t> now, cols, single;
    std::vector<Item> rest;
    for (int todo = nn; todo > 0;) {
      // what cannot wait, then the most urgent ready nodes while they fit in the
      // units that takes (or that all ready ones take, four at most)
      const int tick = (int)out.size();
      now.clear();
      rest.clear();
      int64_t all = 0, used = 0;
      int depth = 1;
      while (!q.empty()) {
        const Item it = q.top();
        q.pop();
        const int64_t c = (int64_t)nodes[it.second].lanes * units(nodes[it.second]);
        all += c;
        if (it.first <= tick) {
          now.push_back(it.second);
          used += c;
          depth = std::max(depth, units(nodes[it.second]));
        } else {
          rest.push_back(it);
        }
      }
      const int64_t wide = 32 * kSoloWarps;
      depth = std::max<int64_t>({(int64_t)depth, (used + wide - 1) / wide, std::min<int64_t>(4, all / wide)});
      for (const Item& it : rest) {
        const int u = units(nodes[it.second]);
        const int64_t c = (int64_t)nodes[it.second].lanes * u;
        if (u <= depth && used + c <= depth * wide * 9 / 10) {
          now.push_back(it.second);
          used += c;
        } else {
          q.push(it);
        }
      }
      // lanes: columns first (their lanes in one warp), then the sums, the longest
      // first, into warps that run as many units anyway
      std::vector<Vec> vecs;
      cols.clear();
      single.clear();
      for (int i : now) (nodes[i].t1 < 0 ? cols : single).push_back(i);
      auto longer = [&](int x, int y) { return units(nodes[x]) > units(nodes[y]); };
      std::stable_sort(cols.begin(), cols.end(), longer);
      std::stable_sort(single.begin(), single.end(), longer);
      size_t open = 0;
      for (int i : cols) {
        const int k = nodes[i].v, d = sc.c_base[k] + sc.c_ulen[k], ll = sc.c_llen[k], u = units(nodes[i]);
        for (int e0 = 0; e0 == 0 || e0 < ll; e0 += 31) {
          const int cnt = 1 + std::min(31, ll - e0);
          size_t x = open;
          while (x < vecs.size() && 32 - (int)vecs[x].lane.size() < cnt) x++;
          if (x == vecs.size()) vecs.emplace_back();
          Vec& w = vecs[x];
          const uint32_t src = (uint32_t)w.lane.size();
          w.col = true;
          w.units = std::max(w.units, u);
          // (a pivot with more L entries than lanes is stored already)
          w.lane.push_back({d, from[d], stop[d], src | SOLO_PIVOT | (ll > 31 ? 0u : SOLO_STORE)});
          for (int e = e0 + 1; e < e0 + cnt; e++)
            w.lane.push_back({d + e, from[d + e], stop[d + e], src | SOLO_SCALE | SOLO_STORE});
          while (open < vecs.size() && vecs[open].lane.size() == 32) open++;
        }
      }
      size_t at = 0;
      for (int i : single) {
        while (at < vecs.size() && vecs[at].lane.size() == 32) at++;
        if (at == vecs.size()) vecs.emplace_back();
        vecs[at].lane.push_back({nodes[i].v, nodes[i].t0, nodes[i].t1, SOLO_STORE});
        vecs[at].units = std::max(vecs[at].units, units(nodes[i]));
      }
      out.push_back(std::move(vecs));
      todo -= (int)now.size();
      for (int i : now)
        for (int s = sptr[i]; s < sptr[i + 1]; s++)
          if (--npred[succ[s]] == 0) q.push({nodes[succ[s]].late, succ[s]});
    }
    for (int k : columns) {  // (for a later launch all of this is done before)
      auto ran = [&](int v) {
        done[v] = -1;
        taken[v] = stop[v] - S.ptr[v];
        stop[v] = S.ptr[v + 1];
      };
      for (int v = sc.c_base[k]; v < sc.c_base[k] + sc.c_ulen[k] + 1 + sc.c_llen[k]; v++) ran(v);
      ran(ns + k);
    }
    return out;
  };

  // ---- a CTA's backward rows, level by level
  std::vector<int32_t> lev(n, 0);
  auto backward = [&](const std::vector<int32_t>& columns, Ticks& out) {
    const size_t base = out.size();
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
      if (out.size() <= base + l) out.resize(base + l + 1);
      std::vector<Vec>& vecs = out[base + l];
      if (vecs.empty()) vecs.emplace_back();
      vecs[0].lane.push_back({k, sc.bw_ptr[k], sc.bw_ptr[k + 1], SOLO_STORE});
    }
    for (size_t t = base; t < out.size(); t++) {
      std::vector<Lane> rows = std::move(out[t][0].lane);
      std::stable_sort(rows.begin(), rows.end(),
                       [](const Lane& x, const Lane& y) { return units_of(x.t1 - x.t0) > units_of(y.t1 - y.t0); });
      out[t].clear();
      for (size_t i = 0; i < rows.size(); i += 32) {
        out[t].emplace_back();
        Vec& w = out[t].back();
        w.lane.assign(rows.begin() + i, rows.begin() + std::min(rows.size(), i + 32));
        w.units = units_of(w.lane[0].t1 - w.lane[0].t0);
      }
    }
  };

  // ---- a CTA's streams; ticks from `back` on are backward rows
  const uint32_t el = (uint32_t)plan.elem;
  std::vector<int32_t> place(zero + 1, -1);  // a value's place in the CTA's
  std::vector<char> in_sol(n, 0);            // rows that an earlier launch stored
  auto streams = [&](const Ticks& ticks, size_t back, int which) {
    SoloCta C;
    // the values it uses, in the order of their numbers; what it writes of them
    // that a later launch reads: all, the rest's CTA only its x
    std::vector<int32_t> used, wrote;
    auto use = [&](int v) {
      if (place[v] < 0) {
        place[v] = 0;
        used.push_back(v);
      }
    };
    for (size_t t = 0; t < ticks.size(); t++)
      for (const Vec& v : ticks[t])
        for (const Lane& s : v.lane) {
          const bool div = t >= back;
          const int to = div ? ns + s.v : s.v;
          use(to);
          if ((s.info & SOLO_STORE) && (which != 2 || div)) wrote.push_back(to);
          if (div) use(sc.diag_slot[s.v]);
          for (int e = s.t0; e < s.t1; e++) {
            use(div ? sc.bw_slot[e] : S.a[e]);
            use(div ? ns + sc.bw_col[e] : second(s.v, e));
          }
        }
    std::sort(used.begin(), used.end());
    std::sort(wrote.begin(), wrote.end());
    wrote.erase(std::unique(wrote.begin(), wrote.end()), wrote.end());
    for (size_t i = 0; i < used.size(); i++) place[used[i]] = (int32_t)i;
    place[zero] = (int32_t)used.size();
    C.load = (int32_t)P.lists.size();
    C.n_load = (int32_t)used.size();
    for (int v : used)
      P.lists.push_back(v < ns ? SOLO_LU | (uint32_t)v : (in_sol[v - ns] ? SOLO_SOL : SOLO_RHS) | (uint32_t)(v - ns));
    if (P.lists.size() & 1) P.lists.push_back(0u);  // (read by pairs)
    C.store = (int32_t)P.lists.size();
    C.n_store = (int32_t)wrote.size();
    for (int v : wrote) {
      P.lists.push_back(v < ns ? SOLO_LU | (uint32_t)v : SOLO_SOL | (uint32_t)(v - ns));
      P.lists.push_back((uint32_t)place[v]);
      if (v >= ns) in_sol[v - ns] = 1;
    }
    P.max_values[which] = std::max(P.max_values[which], C.n_load + 1);
    auto off = [&](int v) { return (uint32_t)place[v] * el; };
    std::vector<std::vector<uint32_t>> w(kSoloWarps);
    std::vector<double> load(kSoloWarps);
    auto flags = [&](std::vector<uint32_t>& x) { return x.end() - kSoloQuads * 4; };
    auto set = [&](std::vector<uint32_t>& x, uint32_t f) {  // onto the last unit's flags
      auto u = flags(x);
      for (int l = 0; l < 32; l++) u[(2 * 32 + l) * 4 + 3] += f;
    };
    auto unit = [&](std::vector<uint32_t>& x) {
      x.resize(x.size() + kSoloQuads * 4, 0u);
      return x.end() - kSoloQuads * 4;
    };
    // a unit without sums
    auto idle = [&](std::vector<uint32_t>& x, uint32_t f) {
      auto u = unit(x);
      for (int l = 0; l < 32; l++)
        for (int i = 0; i < 12; i++)
          u[((i / 4) * 32 + l) * 4 + i % 4] = i < 9 ? off(zero) : i == 9 ? (uint32_t)l : i == 11 ? f : 0u;
    };
    int turn = 0;
    for (size_t t = 0; t < ticks.size(); t++) {
      const bool div = t >= back;
      std::fill(load.begin(), load.end(), 0.0);
      std::vector<const Vec*> order;
      for (const Vec& v : ticks[t]) order.push_back(&v);
      std::stable_sort(order.begin(), order.end(), [](const Vec* a, const Vec* b) { return a->units > b->units; });
      for (const Vec* v : order) {
        // (in turn among the least loaded)
        int b = -1;
        for (int i = 0; i < kSoloWarps; i++) {
          const int c = (turn + i) % kSoloWarps;
          if (b < 0 || load[c] < load[b]) b = c;
        }
        turn = (b + 1) % kSoloWarps;
        load[b] += v->units + (v->col ? 0.5 : 0.0);
        for (int u = 0; u < v->units; u++) {
          auto x = unit(w[b]);
          auto word = [&](int l, int i) -> uint32_t& { return x[((i / 4) * 32 + l) * 4 + i % 4]; };
          const bool last = u + 1 == v->units;
          uint32_t most = 0;
          for (const Lane& s : v->lane)
            most = std::max(most, (uint32_t)std::clamp(s.t1 - s.t0 - u * kSoloTerms, 0, kSoloTerms));
          const uint32_t f = (u > 0 ? SOLO_CIN : 0u) | (last ? 0u : SOLO_COUT) | (v->col && last ? SOLO_COL : 0u) |
                             (div ? SOLO_DIV : 0u) | most << 4;
          for (int l = 0; l < 32; l++) {
            word(l, 0) = off(zero);
            for (int i = 1; i <= 2 * kSoloTerms; i++) word(l, i) = off(zero);
            word(l, 9) = (uint32_t)l;
            word(l, 10) = div ? off(sc.diag_slot[v->lane[0].v]) : 0u;
            word(l, 11) = f;
            if (l >= (int)v->lane.size()) continue;
            const Lane& s = v->lane[l];
            word(l, 0) = off(div ? ns + s.v : s.v);
            if (last)
              word(l, 9) = (s.info & ~SOLO_SRC) |
                           (v->col && (s.info & (SOLO_PIVOT | SOLO_SCALE)) ? s.info & SOLO_SRC : (uint32_t)l);
            if (div) word(l, 10) = off(sc.diag_slot[s.v]);
            for (int i = 0; i < kSoloTerms; i++) {
              const int e = s.t0 + u * kSoloTerms + i;
              if (e >= s.t1) break;
              word(l, 1 + 2 * i) = off(div ? sc.bw_slot[e] : S.a[e]);
              word(l, 2 + 2 * i) = off(div ? ns + sc.bw_col[e] : second(s.v, e));
            }
          }
        }
      }
      if (t + 1 < ticks.size())
        for (auto& x : w) {
          if (x.empty()) idle(x, t >= back ? SOLO_DIV : 0u);
          set(x, 1u << 8);
        }
    }
    for (int i = 0; i < kSoloWarps; i++) {
      idle(w[i], SOLO_END);
      C.stream[i] = (int32_t)(P.words.size() / (kSoloQuads * 4));
      P.words.insert(P.words.end(), w[i].begin(), w[i].end());
    }
    P.launch[which].push_back(C);
    for (int v : used) place[v] = -1;
  };
  std::vector<int32_t> top;
  for (int k = 0; k < n; k++)
    if (stage[k] == 2) top.push_back(k);
  for (auto& m : mid) {
    const Ticks t = forward(m, false);
    streams(t, t.size(), 0);
  }
  if (!mid.empty())
    for (size_t i = 0; i < top.size();) {
      std::vector<int32_t> cols;
      for (; i < top.size() && (int)cols.size() < plan.cols; i++) {
        const int k = top[i], base = sc.c_base[k], len = sc.c_ulen[k] + 1 + sc.c_llen[k];
        bool any = false;
        auto prefix = [&](int v) {
          for (stop[v] = S.ptr[v]; stop[v] < S.ptr[v + 1]; stop[v]++) {
            const int a = S.a[stop[v]], b = S.b[stop[v]];
            if (stage[S.col[a]] > 1 || (v >= ns ? stage[b] > 1 : stop[b] < S.ptr[b + 1])) break;
          }
          any |= stop[v] > S.ptr[v];
        };
        for (int d = 0; d < len; d++) prefix(base + d);
        prefix(ns + k);
        if (any) {
          cols.push_back(k);
        } else {
          for (int d = 0; d < len; d++) stop[base + d] = S.ptr[base + d + 1];
          stop[ns + k] = S.ptr[ns + k + 1];
        }
      }
      if (cols.empty()) continue;
      const Ticks t = forward(cols, true);
      streams(t, t.size(), 1);
    }
  {
    Ticks t = forward(top, false);
    const size_t back = t.size();
    backward(top, t);
    streams(t, back, 2);
  }
  for (auto& m : mid) {
    Ticks t;
    backward(m, t);
    streams(t, 0, 3);
  }
  P.words.insert(P.words.end(), (size_t)kSoloAhead * kSoloQuads * 4, 0u);
  return *std::max_element(P.max_values, P.max_values + 4) <= max_values;
}

std::string run_solo_host(const Schedule& sc, const SoloProgram& P, std::vector<double>& lu,
                          const std::vector<double>& rhs, std::vector<double>& X, bool& singular) {
  const int n = sc.n_u, ns = sc.n_slots, zero = ns + n;
  const Sums S = make_sums(sc);
  singular = false;
  // the values by number, as a CTA's shared memory holds them, and as the batch's
  // memory does; a value's number by its place in the running CTA
  std::vector<double> c(zero + 1, 0.0), mem(zero, 0.0);
  std::vector<char> stored(n, 0), mine(zero + 1, 0);  // rows stored; values the CTA loaded
  std::vector<int32_t> number;
  for (int v = 0; v < ns; v++) mem[v] = lu[v];
  std::vector<int32_t> taken(zero, 0);
  std::vector<char> fin(zero + 1, 0), xdone(n, 0);
  fin[zero] = 1;
  for (int k = 0; k < n; k++) {
    for (int v = sc.c_base[k]; v < sc.c_base[k] + sc.c_ulen[k]; v++) fin[v] = S.ptr[v + 1] == S.ptr[v];
    fin[ns + k] = S.ptr[ns + k + 1] == S.ptr[ns + k];
  }
  // who wrote and read a value last (a lane's sum in a tick), and in which tick,
  // launch and CTA
  std::vector<int64_t> wtick(zero, -1), rtick(zero, -1), wown(zero, -1), rown(zero, -1);
  std::vector<int32_t> wlaunch(zero, -1), rlaunch(zero, -1), wcta(zero, -1), rcta(zero, -1);
  int64_t tick = 0, owner = 0;
  int32_t launch_no = 0, cta = 0;
  std::string err;
  auto fail = [&](const char* s) {
    if (err.empty()) err = s;
    return false;
  };
  auto read = [&](int v, int64_t own) {
    if (v == zero) return true;
    if (!mine[v]) return fail("a value that was not loaded");
    if (wtick[v] == tick && wown[v] != own) return fail("a value read in the tick it is written");
    if (wlaunch[v] == launch_no && wcta[v] != cta) return fail("a value read in the launch another CTA writes it");
    if (rtick[v] != tick) rown[v] = own;
    else if (rown[v] != own) rown[v] = -2;
    rtick[v] = tick;
    if (rlaunch[v] != launch_no) rcta[v] = cta;
    else if (rcta[v] != cta) rcta[v] = -2;
    rlaunch[v] = launch_no;
    return true;
  };
  auto write = [&](int v, int64_t own) {
    if (v == zero) return fail("the zero written");
    if ((wtick[v] == tick && wown[v] != own) || (rtick[v] == tick && rown[v] != own))
      return fail("a value written in the tick another sum uses it");
    if ((wlaunch[v] == launch_no && wcta[v] != cta) || (rlaunch[v] == launch_no && rcta[v] != cta))
      return fail("a value written in the launch another CTA uses it");
    wtick[v] = tick;
    wown[v] = own;
    wlaunch[v] = launch_no;
    wcta[v] = cta;
    return true;
  };
  const size_t nu = P.words.size() / (kSoloQuads * 4);
  const uint32_t el = (uint32_t)P.plan.elem;
  struct Warp {
    size_t at;
    uint32_t bars = 0;
    bool ended = false, open = false, back = false;
    double acc[32];
    int32_t v[32];
    int64_t own[32];
  };
  // a warp up to its next barrier or its end
  auto step = [&](Warp& w) -> bool {
    if (w.bars > 0 && --w.bars > 0) return true;
    if (w.ended) return true;
    for (;;) {
      if (w.at + kSoloAhead >= nu) return fail("a stream runs past the program");
      const uint32_t* u = &P.words[w.at * kSoloQuads * 4];
      auto word = [&](int l, int i) { return u[((i / 4) * 32 + l) * 4 + i % 4]; };
      const uint32_t f = word(0, 11);
      for (int l = 1; l < 32; l++)
        if (word(l, 11) != f) return fail("lanes with different flags");
      w.at++;
      if (f & SOLO_END) {
        w.ended = true;
        return (!w.open && f == SOLO_END) || fail("a sum left open");
      }
      if (w.back && !(f & SOLO_DIV)) return fail("a forward unit after backward ones");
      w.back = (f & SOLO_DIV) != 0;
      {
        if (((f & SOLO_CIN) != 0) != w.open) return fail("a sum carried to another unit");
        double piv[32];
        int32_t pv[32];
        for (int l = 0; l < 32; l++) {
          for (int i = 0; i < 11; i++)
            if (i != 9 && (word(l, i) % el || word(l, i) / el >= number.size())) return fail("a value out of range");
          const int v = number[word(l, 0) / el];
          const bool lives = v != zero;
          if (f & SOLO_CIN) {
            if (v != w.v[l]) return fail("a sum carried to another value");
          } else {
            w.v[l] = v;
            w.own[l] = owner++;
            if (!read(v, w.own[l])) return false;
            w.acc[l] = c[v];
            if (lives && (f & SOLO_DIV) && (v < ns || v == zero || !fin[v])) return fail("x before y is final");
            if ((f & SOLO_DIV) && lives) taken[v] = 0;
          }
          for (int i = 0; i < kSoloTerms; i++) {
            const int a = number[word(l, 1 + 2 * i) / el], b = number[word(l, 2 + 2 * i) / el];
            if (a == zero && b == zero) continue;
            if (!lives || a >= ns || b == zero) return fail("a product out of range");
            if (!read(a, w.own[l]) || !read(b, w.own[l])) return false;
            if (f & SOLO_DIV) {
              const int e = sc.bw_ptr[v - ns] + taken[v]++;
              if (e >= sc.bw_ptr[v - ns + 1] || a != sc.bw_slot[e] || b != ns + sc.bw_col[e])
                return fail("a backward term out of order");
              if (!fin[a] || !xdone[b - ns]) return fail("a backward term before its x");
            } else {
              const int e = S.ptr[v] + taken[v]++;
              if (e >= S.ptr[v + 1] || a != S.a[e] || b != (v >= ns ? ns + S.b[e] : S.b[e]))
                return fail("a product out of order");
              if (!fin[a] || !fin[b]) return fail("a product before its value is final");
            }
            if ((uint32_t)i >= ((f >> 4) & 7u)) return fail("a product that is not run");
            w.acc[l] -= c[a] * c[b];
          }
          if (!(f & SOLO_COUT) && lives != ((word(l, 9) & (SOLO_STORE | SOLO_PIVOT)) != 0)) return fail("a sum that is lost");
          if ((f & SOLO_COUT) && (word(l, 9) & ~SOLO_SRC)) return fail("a sum that ends early");
          piv[l] = w.acc[l];
          pv[l] = v;
        }
        w.open = (f & SOLO_COUT) != 0;
        if (!w.open) {
          for (int l = 0; l < 32; l++) {
            const int v = w.v[l];
            const uint32_t info = word(l, 9);
            const bool whole = v < zero && !(f & SOLO_DIV) && taken[v] == S.ptr[v + 1] - S.ptr[v];
            double out = w.acc[l];
            if (info & (SOLO_PIVOT | SOLO_SCALE)) {
              const int src = (int)(info & SOLO_SRC);
              if (!(f & SOLO_COL) || v >= ns) return fail("a column outside a column unit");
              const int d = sc.diag_slot[S.col[v]];
              if (pv[src] != d || !(word(src, 9) & SOLO_PIVOT)) return fail("an L entry of another column's pivot");
              if (!whole || taken[d] != S.ptr[d + 1] - S.ptr[d]) return fail("a column finished before its sums");
              if (info & SOLO_PIVOT) {
                if (v != d || (info & SOLO_SCALE) || src != l) return fail("a pivot that is none");
                if (out == 0) singular = true;
              } else {
                if (v <= d || v > d + sc.c_llen[S.col[v]]) return fail("an L entry that is none");
                out = out * (1.0 / piv[src]);
              }
            } else if ((f & SOLO_COL) && (int)(info & SOLO_SRC) != l) {
              return fail("a lane with another's pivot");
            }
            if (f & SOLO_DIV) {
              if (!(info & SOLO_STORE)) continue;
              const int k = v - ns;
              const int d = number[word(l, 10) / el];
              if (d != sc.diag_slot[k] || !fin[d]) return fail("a backward row with another pivot");
              if (!read(d, w.own[l])) return false;
              if (taken[v] != sc.bw_ptr[k + 1] - sc.bw_ptr[k]) return fail("an incomplete backward row");
              out = out / c[d];
              if (!std::isfinite(out)) singular = true;
              xdone[k] = 1;
            } else if (info & SOLO_STORE) {
              if (fin[v] && S.ptr[v + 1] > S.ptr[v]) return fail("a final value written again");
            }
            if (info & SOLO_STORE) {
              if (!write(v, w.own[l])) return false;
              c[v] = out;
              if (!(f & SOLO_DIV) && whole) {
                // (a pivot's or an L entry's sum without SOLO_PIVOT / SCALE is raw)
                const bool lower = v < ns && v >= sc.diag_slot[S.col[v]];
                if (!lower || (info & (SOLO_PIVOT | SOLO_SCALE))) fin[v] = 1;
              }
            }
            if ((info & SOLO_PIVOT) && !(info & SOLO_STORE)) fin[v] = 1;  // stored in an earlier tick
          }
        }
      }
      w.bars = f >> 8;
      if (w.bars) return !w.open || fail("a barrier inside a sum");
    }
  };
  for (int L = 0; L < 4; L++) {
    launch_no++;
    for (size_t b = 0; b < P.launch[L].size(); b++) {
      const SoloCta& C = P.launch[L][b];
      cta = (int32_t)b;
      if (C.load < 0 || C.n_load < 0 || C.store < 0 || C.n_store < 0 || (size_t)C.load + C.n_load > P.lists.size() ||
          (size_t)C.store + 2 * (size_t)C.n_store > P.lists.size() || C.n_load + 1 > P.max_values[L])
        return "a list out of range";
      number.clear();
      for (int i = 0; i < C.n_load; i++) {
        const uint32_t x = P.lists[C.load + i], from = x & SOLO_WHERE, e = x & ~SOLO_WHERE;
        if (e >= (uint32_t)(from == SOLO_LU ? ns : n)) return "a loaded value out of range";
        const int v = (int)(from == SOLO_LU ? e : ns + e);
        if (from == SOLO_WHERE || (from != SOLO_LU && (from == SOLO_SOL) != (stored[e] != 0))) return "a row from the wrong place";
        if (mine[v] || (wlaunch[v] == launch_no && wcta[v] != cta)) return "a value loaded in the launch another CTA writes it";
        if (rlaunch[v] != launch_no) rcta[v] = cta;
        else if (rcta[v] != cta) rcta[v] = -2;
        rlaunch[v] = launch_no;
        mine[v] = 1;
        c[v] = from == SOLO_RHS ? rhs[e] : mem[v];
        number.push_back(v);
      }
      number.push_back(zero);
      std::vector<Warp> w;
      for (int i = 0; i < kSoloWarps; i++) {
        Warp x;
        if (C.stream[i] < 0) return "a stream out of range";
        x.at = (size_t)C.stream[i];
        w.push_back(x);
      }
      for (int ended = 0; ended < kSoloWarps;) {
        ended = 0;
        for (auto& x : w) {
          if (!step(x)) return err;
          ended += x.ended;
        }
        if (ended != 0 && ended != kSoloWarps) return "the warps take different numbers of barriers";
        tick++;
      }
      for (int i = 0; i < C.n_store; i++) {
        const uint32_t x = P.lists[C.store + 2 * i], to = x & SOLO_WHERE, e = x & ~SOLO_WHERE, at = P.lists[C.store + 2 * i + 1];
        if ((to != SOLO_LU && to != SOLO_SOL) || e >= (uint32_t)(to == SOLO_LU ? ns : n) || at >= (uint32_t)C.n_load)
          return "a stored value out of range";
        const int v = (int)(to == SOLO_LU ? e : ns + e);
        if (number[at] != v) return "another value's place stored";
        if ((wlaunch[v] == launch_no && wcta[v] != cta) || (rlaunch[v] == launch_no && rcta[v] != cta))
          return "a value stored in the launch another CTA uses it";
        mem[v] = c[v];
        if (v >= ns) stored[e] = 1;
      }
      for (int v : number) mine[v] = 0;
    }
  }
  if (P.launch[2].size() != 1) return "a rest of other than one CTA";
  for (int k = 0; k < n; k++)
    if (!stored[k] || !(mem[ns + k] == c[ns + k] || std::isnan(c[ns + k]))) return "a row of the solution is not stored";
  for (int v = 0; v < zero; v++)
    if (!fin[v]) return "a value is left unfinished";
  for (int k = 0; k < n; k++)
    if (!xdone[k]) return "a row of the solution is left out";
  for (int v = 0; v < ns; v++) lu[v] = c[v];
  X.assign(c.begin() + ns, c.begin() + ns + n);
  return err;
}

}  // namespace gox
