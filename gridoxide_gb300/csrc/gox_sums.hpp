// What the compilers of the refactor's programs share: the sums of a schedule
// and the parts of its elimination forest.
#pragma once
#include <algorithm>
#include <cstdint>
#include <queue>
#include <vector>

#include "gox_engine.hpp"

namespace gox {

// The sums of a schedule: per value its ordered terms.  Values are numbered
// LU slots first, then y (row k at n_slots + k).
struct Sums {
  std::vector<int32_t> ptr, a, b;  // value -> terms
  std::vector<int32_t> col;        // LU slot -> column
};

inline Sums make_sums(const Schedule& sc) {
  Sums s;
  const int n = sc.n_u, ns = sc.n_slots;
  s.ptr.assign((size_t)ns + n + 1, 0);
  s.col.assign(ns, 0);
  for (int k = 0; k < n; k++) {
    const int base = sc.c_base[k];
    for (int d = 0; d < sc.c_ulen[k] + 1 + sc.c_llen[k]; d++) s.col[base + d] = k;
    for (int e = sc.cu_ptr[k]; e < sc.cu_ptr[k + 1]; e++)
      for (int t = sc.cu_dptr[e]; t < sc.cu_dptr[e + 1]; t++) s.ptr[base + sc.cu_dst[t] + 1]++;
    if (sc.fuse_fwd) s.ptr[ns + k + 1] += sc.fw_ptr[k + 1] - sc.fw_ptr[k];
  }
  for (size_t v = 0; v + 1 < s.ptr.size(); v++) s.ptr[v + 1] += s.ptr[v];
  s.a.assign(s.ptr.back(), 0);
  s.b.assign(s.ptr.back(), 0);
  std::vector<int32_t> at(s.ptr.begin(), s.ptr.end() - 1);
  for (int k = 0; k < n; k++) {
    const int base = sc.c_base[k];
    for (int e = sc.cu_ptr[k]; e < sc.cu_ptr[k + 1]; e++) {
      const int j = sc.cu_j[e], l0 = sc.c_base[j] + sc.c_ulen[j] + 1;
      for (int t = sc.cu_dptr[e]; t < sc.cu_dptr[e + 1]; t++) {
        const int v = base + sc.cu_dst[t];
        s.a[at[v]] = l0 + (t - sc.cu_dptr[e]);
        s.b[at[v]++] = base + (e - sc.cu_ptr[k]);
      }
    }
    if (sc.fuse_fwd)
      for (int t = sc.fw_ptr[k]; t < sc.fw_ptr[k + 1]; t++) {
        s.a[at[ns + k]] = sc.fw_slot[t];
        s.b[at[ns + k]++] = sc.fw_col[t];
      }
  }
  return s;
}

// Columns in stages, those of a stage in independent parts.
struct Parts {
  const Schedule& sc;
  std::vector<char> stage;      // per column: 0 bottom, 1 mid, 2 top
  std::vector<double> cost;     // rough cycles of a column on one warp
  std::vector<int32_t> parent;  // union-find of a stage's parts
  std::vector<double> sum;      // cost of a root's part

  Parts(const Schedule& sched, const Sums& S)
      : sc(sched), stage(sched.n_u, 2), cost(sched.n_u, 0.0), parent(sched.n_u), sum(sched.n_u, 0.0) {
    for (int k = 0; k < sc.n_u; k++) {
      cost[k] = 300.0 + 12.0 * (sc.c_ulen[k] + 1 + sc.c_llen[k]);
      for (int e = sc.cu_ptr[k]; e < sc.cu_ptr[k + 1]; e++) cost[k] += 40.0 + 8.0 * (sc.cu_dptr[e + 1] - sc.cu_dptr[e]);
      if (sc.fuse_fwd) cost[k] += 8.0 * (S.ptr[sc.n_slots + k + 1] - S.ptr[sc.n_slots + k]);
    }
  }
  double cost_from(char st) const {
    double c = 0;
    for (int k = 0; k < sc.n_u; k++)
      if (stage[k] >= st) c += cost[k];
    return c;
  }
  int find(int k) {
    while (parent[k] != k) k = parent[k] = parent[parent[k]];
    return k;
  }
  // columns into stage st: those whose dependences are in earlier stages or in a
  // part of theirs, as long as their part costs no more than cap
  void grow(char st, double cap) {
    std::vector<int32_t> roots;
    for (int k = 0; k < sc.n_u; k++) {
      if (stage[k] < st) continue;
      bool ok = true;
      roots.clear();
      double c = cost[k];
      auto dep = [&](int j) {
        if (stage[j] < st) return;
        if (stage[j] > st) {
          ok = false;
          return;
        }
        const int r = find(j);
        if (std::find(roots.begin(), roots.end(), r) == roots.end()) {
          roots.push_back(r);
          c += sum[r];
        }
      };
      for (int e = sc.cu_ptr[k]; ok && e < sc.cu_ptr[k + 1]; e++) dep(sc.cu_j[e]);
      if (sc.fuse_fwd)
        for (int t = sc.fw_ptr[k]; ok && t < sc.fw_ptr[k + 1]; t++) dep(sc.fw_col[t]);
      if (!ok || c > cap) continue;
      stage[k] = st;
      parent[k] = k;
      for (int r : roots) parent[r] = k;
      sum[k] = c;
    }
  }
  // a stage's parts to its workers, largest first onto the least loaded one
  std::vector<std::vector<int32_t>> deal(char st, int workers) {
    std::vector<std::vector<int32_t>> members(sc.n_u), out(workers);
    std::vector<int32_t> roots;
    for (int k = 0; k < sc.n_u; k++)
      if (stage[k] == st) {
        const int r = find(k);
        members[r].push_back(k);
        if (r == k) roots.push_back(k);
      }
    std::stable_sort(roots.begin(), roots.end(), [&](int x, int y) { return sum[x] > sum[y]; });
    std::priority_queue<std::pair<double, int>, std::vector<std::pair<double, int>>, std::greater<>> q;
    for (int b = 0; b < workers; b++) q.push({0.0, b});
    for (int r : roots) {
      auto [c, b] = q.top();
      q.pop();
      out[b].insert(out[b].end(), members[r].begin(), members[r].end());
      q.push({c + sum[r], b});
    }
    return out;
  }
};

}  // namespace gox
