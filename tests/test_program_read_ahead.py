"""CPU: the checking interpreters of the dot and solo programs allow no read
past a program's words.

The kernels fetch a stream's words ahead of the unit they run.  A program as
compiled must pass; one whose words end a chunk (dot) or a unit (solo) earlier,
so that the fetch of its last stream would pass the end, must be refused."""
import os
import subprocess

_MAIN = r"""
#include <cstdio>
#include "gox_dot.hpp"
#include "gox_solo.hpp"
using namespace gox;
int main() {
  const int n = 37;
  std::vector<int32_t> r, c;
  std::vector<double> v;
  for (int i = 0; i < n; i++)
    for (int j : {i, i + 1, i - 1, (7 * i) % n}) {
      if (j < 0 || j >= n) continue;
      r.push_back(i);
      c.push_back(j);
      v.push_back(i == j ? 9.0 : 1.0);
    }
  const Csc A = build_csc(n, (int)r.size(), r.data(), c.data());
  const Symbolic S = klu_analyze(n, A.p.data(), A.i.data());
  std::vector<double> packed(A.nnz(), 0.0);
  for (size_t e = 0; e < v.size(); e++) packed[A.slot_of[e]] += v[e];
  Numeric N;
  if (klu_factor(A, packed.data(), S, 0.001, N)) return 2;
  Schedule sc;
  build_schedule(nullptr, A, S, N, sc);
  bool sing = false;
  std::vector<double> X;
  auto dot = [&](const DotProgram& p) {
    std::vector<double> lu(sc.n_slots, 1.0), rhs(n, 0.0);
    return run_dot_host(sc, p, lu, rhs, X, sing);
  };
  auto solo = [&](const SoloProgram& p) {
    std::vector<double> lu(sc.n_slots, 1.0), rhs(n, 0.0);
    return run_solo_host(sc, p, lu, rhs, X, sing);
  };
  for (int elem : {4, 8}) {
    DotProgram p;
    build_dot(sc, dot_default(sc, elem, 1), p);
    std::printf("dot %s|", dot(p).c_str());
    p.words.resize(p.words.size() - 4 * kDotChunk);
    std::printf("%s\n", dot(p).c_str());
    SoloProgram q;
    if (!build_solo_default(sc, elem, true, q)) return 3;
    std::printf("solo %s|", solo(q).c_str());
    q.words.resize(q.words.size() - kSoloQuads * 4);
    std::printf("%s\n", solo(q).c_str());
  }
  return 0;
}
"""


def test_interpreters_refuse_a_read_past_the_words(gox, tmp_path):
    from gridoxide_gb300 import build as gb
    objs = []
    os.makedirs(gb.OBJ, exist_ok=True)
    for s in ("gox_symbolic.cpp", "gox_engine.cpp", "gox_dot.cpp", "gox_solo.cpp"):
        o = os.path.join(gb.OBJ, s + ".o")
        objs.append(o if os.path.exists(o) else gb._compile(s, gb._nvcc(), []))
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(_MAIN)
    subprocess.run(["g++", "-std=c++17", "-I", gb.CSRC, str(src)] + objs + ["-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.splitlines()
    assert out == ["dot |a stream runs past the program", "solo |a stream runs past the program"] * 2
