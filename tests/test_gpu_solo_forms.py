"""GPU: the solo programs over every form of a solve.

Few scenarios run the Newton loop in one launch (one CTA per scenario) or the
solo programs of several CTAs from the host's loop.  Each form of a solve must
give the stream plans' results bit for bit: outages, voltage-dependent loads,
both, a start point per scenario, a history, budgets that run out, the longest
budget of the one launch and one more, loads too heavy to converge, a start
that makes the Jacobian infinite.  A child process loads a plan cache that
names one dot plan for every key, so that the solo programs are built whatever
was faster; the launches show which program ran."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_CHILD = r"""
import sys
root, prec, n, b, bins, mid = sys.argv[1], *[int(x) for x in sys.argv[2:]]
sys.path.insert(0, root)
import numpy as np
import gridoxide_gb300 as gox
from gridoxide_gb300 import grids as G
from gridoxide_gb300 import solver as S
g = G.family_grid(n, 3)
yb = G.build_ybus(g)
S.set_autotune(False)
streams = gox.Topology(yb, g.bus_type)
assert streams.prepare(g.p_spec, g.q_spec, g.vm, g.va)
p, q = G.load_scenarios(g, b, 0.15, b)
rng = np.random.default_rng(n)
out = G.outage_deltas(g, yb, rng.choice(np.flatnonzero(~G.bridges(g)), b))
load = 0.1 * (g.load_p + 1j * g.load_q)
zips = [-rng.uniform(0, 1, n) * load, -rng.uniform(0, 1, n) * load]
vm = np.repeat(g.vm[None], b, 0)
va = np.repeat(g.va[None], b, 0) + rng.normal(0, 0.01, (b, n))
zero = vm.copy()
zero[-1] = 0.0
streams.solve(p, q, g.vm, g.va, precision=prec)
S.set_autotune(True)
topo = gox.Topology(yb, g.bus_type)
assert topo.prepare(g.p_spec, g.q_spec, g.vm, g.va)
first = topo.solve(p, q, g.vm, g.va, precision=prec)
dot_launches = topo.last_launches()
for _ in range(2):
    r = topo.solve(p, q, g.vm, g.va, precision=prec)
assert topo.tuning(prec)["chunk_words"] == 128
one_launch = mid == 0
if not one_launch:  # four launches per refactor in place of a dot program's eight
    assert topo.last_fallbacks() == 0
    assert dot_launches - topo.last_launches() == 4 * (int(r.iterations.max()) - 1)
forms = dict(plain=(p, q, g.vm, g.va, {}), outage=(p, q, g.vm, g.va, dict(outage=out)),
             rows=(p, q, vm, va, {}), rows_outage=(p, q, vm, va, dict(outage=out, history=True)),
             heavy=(6 * p, 6 * q, g.vm, g.va, dict(max_iter=12, history=True)),
             infinite=(p, q, zero, va, dict(history=True)))
for it in (1, 2, 3, 64, 65):
    forms[f"budget{it}"] = (p, q, g.vm, g.va, dict(max_iter=it, history=True, outage=out))
ended = set()
for terms in (False, True):
    for t in (streams, topo):
        t.set_zip(*zips) if terms else t.set_zip()
    for name, (fp, fq, fvm, fva, kw) in forms.items():
        ref = streams.solve(fp, fq, fvm, fva, precision=prec, **kw)
        r = topo.solve(fp, fq, fvm, fva, precision=prec, **kw)
        if one_launch and topo.last_fallbacks() == 0:
            assert (topo.last_launches() <= 11) == (name != "budget65"), (name, topo.last_launches())
        ended |= set(r.status.tolist())
        for k in ("voltage_mag", "voltage_ang", "iterations", "status", "max_mismatch", "history"):
            if getattr(ref, k) is not None:
                np.testing.assert_array_equal(getattr(ref, k), getattr(r, k), err_msg=f"{n} {terms} {name} {k}")
assert ended >= {gox.GOX_CONVERGED, gox.GOX_MAX_ITERATIONS}, ended
print("same", sorted(ended))
"""


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,b,bins,mid", [(20, 1, 0, 0), (119, 33, 0, 0), (119, 600, 0, 0), (2003, 9, 64, 8)])
def test_solo_forms_equal_streams(tmp_path, precision, n, b, bins, mid):
    """precision: 0 mixed, 1 FP64 (the cache file's numbering)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    sys.path.insert(0, root)
    import gridoxide_gb300 as gox
    cache = tmp_path / "tune.txt"
    with open(cache, "w") as f:
        for bb in range(0, 25):
            for fill in range(0, 60):
                for gb in range(5):
                    f.write(f"gox-tune-3 {precision} {bb} {fill} {gb} {16 if precision else 32} 128 {mid} {bins}\n")
    prec = (gox.GOX_PRECISION_MIXED, gox.GOX_PRECISION_FP64)[precision]
    out = subprocess.run([sys.executable, "-c", _CHILD, root, str(int(prec)), str(n), str(b), str(bins), str(mid)],
                         env=dict(os.environ, GOX_TUNE_CACHE=str(cache)), capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-3000:]
    assert out.stdout.startswith("same")
