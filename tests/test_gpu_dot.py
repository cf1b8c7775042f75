"""GPU: the refactor's dot-product programs.

A program runs the sums of the stream plans on other warps and in other
pieces, each sum's own products in the same order: batched solves must equal
the stream plans' bit for bit.  A child process loads a plan cache that names
one dot plan for every key, so the plan is used whatever it would have
measured.  The sizes are those where a program changes shape: grids of a few
buses, without and with bins, sums that end on and beside a unit's eight
products, one scenario, one more than a group, a ragged third group.

The linear-solver entry runs a program on any matrix: order one, diagonal,
dense (sums of every length up to the order), and several BTF blocks with
entries between them (no substitutions in the program)."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_CHILD = r"""
import sys
root, prec, warps, bins, mid = sys.argv[1], *[int(x) for x in sys.argv[2:6]]
sys.path.insert(0, root)
import numpy as np
import gridoxide_gb300 as gox
from gridoxide_gb300 import grids as G
from gridoxide_gb300 import solver as S
for n in [int(x) for x in sys.argv[6:]]:
    g = G.family_grid(n, 3)
    yb = G.build_ybus(g)
    topo = {}
    for plan in ("streams", "dot"):
        S.set_autotune(plan == "dot")
        topo[plan] = gox.Topology(yb, g.bus_type)
        assert topo[plan].prepare(g.p_spec, g.q_spec, g.vm, g.va)
        for b in (1, 33, 70) + ((1700,) if n <= 131 else ()):
            p, q = G.load_scenarios(g, b, 0.15, b)
            r = topo[plan].solve(p, q, g.vm, g.va, precision=prec)
            if plan == "streams":
                topo[b] = r
                continue
            for k in ("voltage_mag", "voltage_ang", "iterations", "status", "max_mismatch"):
                np.testing.assert_array_equal(getattr(topo[b], k), getattr(r, k), err_msg=f"{n} {b} {k}")
    tu = topo["dot"].tuning(prec)
    assert (tu["source"], tu["warps"], tu["chunk_words"], tu["wide_levels"], tu["wide_phases"]) == (
        "cached", warps, 128, bins, mid), (n, tu)
print("same")
"""


@pytest.mark.parametrize("precision,warps,bins,mid,sizes", [
    (0, 32, 0, 0, (3, 5, 9, 30, 119)), (0, 16, 32, 0, (131, 300)), (0, 32, 64, 0, (700,)),
    (1, 16, 0, 0, (3, 5, 9, 30, 119)), (1, 16, 32, 0, (131, 300)), (1, 16, 64, 0, (700,)),
    (0, 32, 0, 3, (119, 131)), (0, 32, 64, 8, (700,)), (0, 32, 32, 16, (300,)),
    (1, 16, 0, 3, (119, 131)), (1, 16, 64, 8, (700,)), (1, 16, 32, 4, (300,))])
def test_dot_plan_equals_streams(tmp_path, precision, warps, bins, mid, sizes):
    """precision: 0 mixed, 1 FP64 (the cache file's numbering); mid: CTAs of the
    mid stage.  54 groups run the program for many groups."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    sys.path.insert(0, root)
    import gridoxide_gb300 as gox
    cache = tmp_path / "tune.txt"
    with open(cache, "w") as f:
        for bb in range(0, 25):
            for fill in range(0, 60):
                for gb in range(5):
                    f.write(f"gox-tune-3 {precision} {bb} {fill} {gb} {warps} 128 {mid} {bins}\n")
    prec = (gox.GOX_PRECISION_MIXED, gox.GOX_PRECISION_FP64)[precision]
    out = subprocess.run([sys.executable, "-c", _CHILD, root, str(int(prec)), str(warps), str(bins), str(mid)] +
                         [str(n) for n in sizes], env=dict(os.environ, GOX_TUNE_CACHE=str(cache)),
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-3000:]
    assert out.stdout.split()[-1] == "same"


def _blocks(rng):
    """Two dominant blocks with entries above them (BTF: two blocks)."""
    a = np.zeros((23, 23))
    a[:9, :9] = rng.uniform(-1, 1, (9, 9))
    a[9:, 9:] = rng.uniform(-1, 1, (14, 14))
    a[:9, 9:] = rng.uniform(-1, 1, (9, 14)) * (rng.uniform(size=(9, 14)) < 0.3)
    return a


@pytest.mark.parametrize("kind", ["one", "diagonal", "dense8", "dense9", "dense40", "blocks"])
def test_linear_solver_matrices(gox, kind):
    rng = np.random.default_rng(5)
    a = {"one": lambda: np.array([[0.7]]), "diagonal": lambda: np.diag(rng.uniform(1, 2, 17)),
         "dense8": lambda: rng.uniform(-1, 1, (8, 8)), "dense9": lambda: rng.uniform(-1, 1, (9, 9)),
         "dense40": lambda: rng.uniform(-1, 1, (40, 40)), "blocks": lambda: _blocks(rng)}[kind]()
    n = a.shape[0]
    a += np.diag(np.sign(np.diag(a)) * np.abs(a).sum(1))  # row dominant: growth at most 2
    rows, cols = np.nonzero(a)
    s = gox.Gb300LinearSolver.new(n, list(zip(rows.tolist(), cols.tolist(), a[rows, cols].tolist())))
    for _ in range(2):
        v = a[rows, cols] * rng.uniform(0.9, 1.1, rows.size)
        m = np.zeros((n, n))
        m[rows, cols] = v
        b = rng.uniform(-1, 1, n)
        x = s.factor_and_solve_values(v, b)
        # backward error of Gaussian elimination without growth: 3 n u |A||x|
        bound = 8 * n * 2.0 ** -53 * (np.abs(m).sum(1).max() * np.abs(x).max() + np.abs(b).max())
        assert np.abs(m @ x - b).max() <= bound
        np.testing.assert_array_equal(s.factor_and_solve_values_static(v, b), x)
