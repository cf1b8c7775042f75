"""GPU: the dot programs at few scenarios, and a start point shared by one.

A topology with a cached dot plan runs the dot program in its first solve and
solo programs in later ones, so each batch here is the first of a topology of
its own: one group, one more than a group, a ragged third group.  The results
must be the stream plans' bit for bit; the same topology's later solves, which
need fewer launches, show that it was the dot program.

A start point that all scenarios share is expanded once per bus; for one
scenario the general path is what a batch of two with a start row each runs."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_CHILD = r"""
import sys
root, prec = sys.argv[1], int(sys.argv[2])
sys.path.insert(0, root)
import numpy as np
import gridoxide_gb300 as gox
from gridoxide_gb300 import grids as G
from gridoxide_gb300 import solver as S
for n in [int(x) for x in sys.argv[3:]]:
    g = G.family_grid(n, 3)
    yb = G.build_ybus(g)
    S.set_autotune(False)
    streams = gox.Topology(yb, g.bus_type)
    assert streams.prepare(g.p_spec, g.q_spec, g.vm, g.va)
    streams.solve(g.p_spec, g.q_spec, g.vm, g.va, precision=prec)
    S.set_autotune(True)
    for b in (1, 33, 70):
        p, q = G.load_scenarios(g, b, 0.15, b)
        ref = streams.solve(p, q, g.vm, g.va, precision=prec)
        topo = gox.Topology(yb, g.bus_type)
        assert topo.prepare(g.p_spec, g.q_spec, g.vm, g.va)
        first = topo.solve(p, q, g.vm, g.va, precision=prec)
        launches, fallbacks = topo.last_launches(), topo.last_fallbacks()
        assert topo.tuning(prec)["chunk_words"] == 128 and topo.tuning(prec)["source"] == "cached"
        for _ in range(3):
            later = topo.solve(p, q, g.vm, g.va, precision=prec)
        assert fallbacks > 0 or topo.last_launches() < launches, (n, b, launches, topo.last_launches())
        for k in ("voltage_mag", "voltage_ang", "iterations", "status", "max_mismatch"):
            np.testing.assert_array_equal(getattr(ref, k), getattr(first, k), err_msg=f"{n} {b} {k}")
            np.testing.assert_array_equal(getattr(ref, k), getattr(later, k), err_msg=f"later {n} {b} {k}")
print("same")
"""


@pytest.mark.parametrize("precision,bins,mid,sizes", [
    (0, 0, 0, (3, 9, 119)), (0, 32, 0, (131, 300)), (0, 64, 8, (700,)),
    (1, 0, 0, (3, 9, 119)), (1, 32, 0, (131, 300)), (1, 64, 8, (700,))])
def test_dot_programs_of_few_groups(tmp_path, precision, bins, mid, sizes):
    """precision: 0 mixed, 1 FP64 (the cache file's numbering)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    sys.path.insert(0, root)
    import gridoxide_gb300 as gox
    cache = tmp_path / "tune.txt"
    cache.write_text("".join(f"gox-tune-3 {precision} {bus} {fill} {groups} {16 if precision else 32} 128 {mid} {bins}\n"
                             for bus in range(25) for fill in range(60) for groups in range(5)))
    prec = (gox.GOX_PRECISION_MIXED, gox.GOX_PRECISION_FP64)[precision]
    out = subprocess.run([sys.executable, "-c", _CHILD, root, str(int(prec))] + [str(n) for n in sizes],
                         env=dict(os.environ, GOX_TUNE_CACHE=str(cache)), capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-3000:]
    assert out.stdout.split()[-1] == "same"


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_shared_start_of_one_scenario(gox, precision):
    from gridoxide_gb300 import grids as G
    prec = gox.GOX_PRECISION_MIXED if precision == "mixed" else gox.GOX_PRECISION_FP64
    g = G.family_grid(4001, 3)  # from 4,000 buses on one scenario takes the shared start's path
    topo = gox.Topology(G.build_ybus(g), g.bus_type)
    assert topo.prepare(g.p_spec, g.q_spec, g.vm, g.va)
    p, q = G.load_scenarios(g, 1, 0.1, 5)
    va = g.va + np.random.default_rng(4).normal(0.0, 0.01, g.n_bus)
    for _ in range(3):  # (the tuning and the solo programs are over)
        two = topo.solve(np.repeat(p, 2, 0), np.repeat(q, 2, 0), np.repeat(g.vm[None], 2, 0),
                         np.repeat(va[None], 2, 0), precision=prec)
    two_launches = topo.last_launches()
    one = topo.solve(p, q, g.vm, va, precision=prec)
    for k in ("voltage_mag", "voltage_ang", "iterations", "status", "max_mismatch"):
        np.testing.assert_array_equal(getattr(two, k)[:1], getattr(one, k), err_msg=k)
        np.testing.assert_array_equal(getattr(two, k)[1:], getattr(one, k), err_msg=k)
    assert topo.last_launches() == two_launches + 1  # the shared start's kernel
