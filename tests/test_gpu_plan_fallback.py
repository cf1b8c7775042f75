"""GPU: a topology whose dot or solo programs cannot be had runs without them.

A second library is linked from the build's own objects with one of the
program compilers, or its checking interpreter, replaced by one that fails.
Every call that would use its programs must still be answered, with the
results that the stream plans give: a topology with a cached dot plan, one
that times its plans, batches of the other kind than the one it was tuned on,
Q-limit variants (whose programs are not timed), the linear guess, the linear
solver."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_FAIL = {
    "build_dot": ("void", "const Schedule&, const DotPlan&, DotProgram&", "throw std::runtime_error(\"a test's\");"),
    "build_solo_default": ("bool", "const Schedule&, int, bool, SoloProgram&", "throw std::runtime_error(\"a test's\");"),
    "run_dot_host": ("std::string", "const Schedule&, const DotProgram&, std::vector<double>&, const std::vector<double>&, "
                     "std::vector<double>&, bool&", "return \"a test's\";"),
    "run_solo_host": ("std::string", "const Schedule&, const SoloProgram&, std::vector<double>&, "
                      "const std::vector<double>&, std::vector<double>&, bool&", "return \"a test's\";"),
}

_CHILD = r"""
import sys
root, lib, cached, fails = sys.argv[1], sys.argv[2], sys.argv[3] == "1", sys.argv[4]
sys.path.insert(0, root)
import numpy as np
from gridoxide_gb300 import _lib
_lib.LIB_PATH = lib
import gridoxide_gb300 as gox
from gridoxide_gb300 import grids as G
from gridoxide_gb300 import solver as S
FIELDS = ("voltage_mag", "voltage_ang", "iterations", "status", "max_mismatch")
def same(a, b, what):
    for k in FIELDS:
        np.testing.assert_array_equal(getattr(a, k), getattr(b, k), err_msg=f"{what} {k}")
g = G.family_grid(119, 3)
yb = G.build_ybus(g)
for prec in (gox.GOX_PRECISION_MIXED, gox.GOX_PRECISION_FP64):
    S.set_autotune(False)
    ref = gox.Topology(yb, g.bus_type)
    assert ref.prepare(g.p_spec, g.q_spec, g.vm, g.va)
    ref.solve(g.p_spec, g.q_spec, g.vm, g.va, precision=prec)
    S.set_autotune(True)
    topo = gox.Topology(yb, g.bus_type)
    assert topo.prepare(g.p_spec, g.q_spec, g.vm, g.va)
    for b in (1, 1, 1, 33, 1700, 1700, 1):
        p, q = G.load_scenarios(g, b, 0.15, b)
        same(topo.solve(p, q, g.vm, g.va, precision=prec), ref.solve(p, q, g.vm, g.va, precision=prec), b)
    # (a cached dot plan is used where only the solo programs fail)
    assert (topo.tuning(prec)["chunk_words"] == 128) == ("solo" in fails) or not cached
    scaled = gox.Topology(yb, g.bus_type)
    scaled.set_initial_guess("linear")
    for _ in range(3):
        r = scaled.solve_scaled(np.array([0.9, 1.0, 1.1]), g.p_spec, g.q_spec, g.vm, g.va, precision=prec)
    assert (r.status == gox.GOX_CONVERGED).all()
    p, q = G.load_scenarios(g, 6, 0.15, 5)
    base = ref.solve(p, q, g.vm, g.va, precision=gox.GOX_PRECISION_FP64)
    v = base.voltage_mag * np.exp(1j * base.voltage_ang)
    y = np.zeros((g.n_bus, g.n_bus), complex)
    y[np.repeat(np.arange(g.n_bus), np.diff(yb.indptr)), yb.indices] = yb.re + 1j * yb.im
    pv = np.flatnonzero(g.bus_type == G.BUS_PV)[:2]
    hi = np.full(g.n_bus, np.inf)
    hi[pv] = np.median((v * np.conj(v @ y.T)).imag[:, pv], axis=0)
    res, sw, _ = gox.Topology(yb, g.bus_type).solve_qlim(p, q, g.vm, g.va, np.full(g.n_bus, -np.inf), hi,
                                                         precision=prec)
    assert sw.any() and (res.status == gox.GOX_CONVERGED).all()
a = np.diag(np.full(30, 4.0)) + np.diag(np.ones(29), 1) + np.diag(np.ones(29), -1)
rows, cols = np.nonzero(a)
s = gox.Gb300LinearSolver.new(30, list(zip(rows.tolist(), cols.tolist(), a[rows, cols].tolist())))
rhs = np.arange(30.0)
assert np.abs(a @ s.factor_and_solve_values(a[rows, cols], rhs) - rhs).max() < 1e-12
print("answered")
"""


def _failing_library(gb, fails, tmp_path):
    """The build's objects linked with `fails` in place of the function of that name."""
    objs = [os.path.join(gb.OBJ, s + ".o") for s in gb.SOURCES]
    if not all(os.path.exists(o) for o in objs):
        gb.build(force=True)
    calls = subprocess.run(["nm", os.path.join(gb.OBJ, "gox_api.cu.o")], check=True, capture_output=True, text=True)
    name = next(x.split()[-1] for x in calls.stdout.splitlines() if " U " in x and f"{len(fails)}{fails}" in x)
    ret, args, body = _FAIL[fails]
    src, obj, lib = tmp_path / "fails.cpp", tmp_path / "fails.o", tmp_path / "libfails.so"
    src.write_text('#include <stdexcept>\n#include "gox_dot.hpp"\n#include "gox_solo.hpp"\nnamespace gox {\n'
                   f'{ret} fails({args}) asm("__wrap_{name}");\n{ret} fails({args}) {{ {body} }}\n}}\n')
    subprocess.run(["g++", "-c", "-fPIC", "-std=c++17", "-I", gb.CSRC, str(src), "-o", str(obj)], check=True)
    subprocess.run([gb._nvcc(), "-shared", "-o", str(lib)] + objs + [str(obj)] + gb.ARCH +
                   ["-Xlinker", f"--wrap={name}", "-lcudart_static", "-lrt", "-lpthread", "-ldl"], check=True)
    return str(lib)


@pytest.mark.parametrize("fails", sorted(_FAIL))
@pytest.mark.parametrize("cached", [True, False])
def test_programs_that_fail_are_not_used(gox, tmp_path, fails, cached):
    from gridoxide_gb300 import build as gb
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    lib = _failing_library(gb, fails, tmp_path)
    env = dict(os.environ)
    env.pop("GOX_TUNE_CACHE", None)
    if cached:
        cache = tmp_path / "tune.txt"
        cache.write_text("".join(f"gox-tune-3 {pr} {bus} {fill} {groups} {16 if pr else 32} 128 0 0\n"
                                 for pr in (0, 1) for bus in range(25) for fill in range(60) for groups in range(5)))
        env["GOX_TUNE_CACHE"] = str(cache)
    out = subprocess.run([sys.executable, "-c", _CHILD, root, lib, str(int(cached)), fails], env=env,
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-3000:]
    assert out.stdout.split()[-1] == "answered"
    assert "a test's" in out.stderr  # it was asked
