"""CPU: solo programs are compiled only where they can run.

A schedule that no plan fits is left without being scheduled (20,000 buses in
FP64: less time than its dot program takes), and solo_most, which decides
whether a batch is worth compiling for, never lies below the scenarios that a
compiled program runs, from a few unknowns to several CTAs."""
import os
import subprocess

import numpy as np

from gridoxide_gb300 import grids as G

_MAIN = r"""
#include <chrono>
#include <cstdio>
#include "gox_dot.hpp"
#include "gox_solo.hpp"
using namespace gox;
int main(int, char** argv) {
  FILE* f = std::fopen(argv[1], "rb");
  int32_t n[2];
  if (std::fread(n, 4, 2, f) != 2) return 1;
  std::vector<int32_t> r(n[1]), c(n[1]);
  if (std::fread(r.data(), 4, n[1], f) != (size_t)n[1] || std::fread(c.data(), 4, n[1], f) != (size_t)n[1]) return 1;
  const Csc A = build_csc(n[0], n[1], r.data(), c.data());
  const Symbolic S = klu_analyze(n[0], A.p.data(), A.i.data());
  std::vector<double> packed(A.nnz(), -1.0);
  for (int e = 0; e < n[1]; e++)
    if (r[e] == c[e]) packed[A.slot_of[e]] = 1000.0;
  Numeric N;
  if (klu_factor(A, packed.data(), S, 0.001, N)) return 2;
  Schedule sc;
  build_schedule(nullptr, A, S, N, sc);
  for (int elem : {4, 8}) {
    using clk = std::chrono::steady_clock;
    const auto t0 = clk::now();
    DotProgram d;
    build_dot(sc, dot_default(sc, elem, 1), d);
    const auto t1 = clk::now();
    SoloProgram p;
    const bool wide = build_solo_default(sc, elem, true, p);
    const double solo = std::chrono::duration<double>(clk::now() - t1).count();
    int most = wide ? solo_scenarios(p, kSoloDepth) : 0;
    if (build_solo_default(sc, elem, false, p)) most = std::max(most, solo_scenarios(p, kSoloDepth));
    std::printf("%d %d %d %d\n", (int)wide, most, solo_most(sc, elem),
                (int)(solo < std::chrono::duration<double>(t1 - t0).count()));
  }
  return 0;
}
"""


def _pattern(path, n, seed):
    """The Y-bus pattern of a grid, twice in each direction: the pattern of [theta; |V|] by [P; Q]."""
    yb = G.build_ybus(G.family_grid(n, seed))
    i, k = np.repeat(np.arange(n), np.diff(yb.indptr)), yb.indices.astype(np.int64)
    rows = np.concatenate([i, i, i + n, i + n]).astype(np.int32)
    cols = np.concatenate([k, k + n, k, k + n]).astype(np.int32)
    with open(path, "wb") as f:
        np.array([2 * n, rows.size], np.int32).tofile(f)
        rows.tofile(f)
        cols.tofile(f)


def test_solo_programs_only_where_they_run(gox, tmp_path):
    from gridoxide_gb300 import build as gb
    objs = []
    os.makedirs(gb.OBJ, exist_ok=True)
    for s in ("gox_symbolic.cpp", "gox_engine.cpp", "gox_dot.cpp", "gox_solo.cpp"):
        o = os.path.join(gb.OBJ, s + ".o")
        objs.append(o if os.path.exists(o) else gb._compile(s, gb._nvcc(), []))
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(_MAIN)
    subprocess.run(["g++", "-std=c++17", "-I", gb.CSRC, str(src)] + objs + ["-o", str(exe)], check=True)
    for n in (3, 20, 119, 300, 2003, 20000):
        _pattern(tmp_path / "a.bin", n, 3)
        out = subprocess.run([str(exe), str(tmp_path / "a.bin")], check=True, capture_output=True, text=True, timeout=120)
        for elem, line in zip((4, 8), out.stdout.splitlines()):
            wide, runs, most, quick = [int(x) for x in line.split()]
            assert wide == (n < 20000 or elem == 4), (n, elem)
            assert runs <= most, (n, elem)
            assert wide or quick, (n, elem)  # nothing was compiled in vain
            assert n != 2003 or most < 999  # nor is it for a batch that none runs
