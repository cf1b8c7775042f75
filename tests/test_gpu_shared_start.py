"""GPU: one start point for all scenarios against the same start repeated.

From 4,000 buses x groups on, a shared start's trigonometry and currents are
computed once per bus.  The same start given as one row per scenario takes the
general kernels: every output must be the same bits, with per-scenario outages
and with voltage-dependent loads too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("form", ["plain", "outage", "zip"])
@pytest.mark.parametrize("n,b", [(119, 1057), (1000, 97), (2003, 33), (4001, 1)])
def test_shared_start_equals_rows(n, b, form, precision):
    import gridoxide_gb300 as gox
    from gridoxide_gb300 import grids as G

    g = G.family_grid(n, 3)
    yb = G.build_ybus(g)
    topo = gox.Topology(yb, g.bus_type)
    prec = gox.GOX_PRECISION_MIXED if precision == "mixed" else gox.GOX_PRECISION_FP64
    vm, va = g.vm.copy(), g.va + 1e-3 * (np.arange(n) % 13)  # angles that are not zero
    assert n * ((b + 31) // 32) >= 4000
    p, q = G.load_scenarios(g, b, 0.1, b)
    out = None
    if form == "outage":
        br = np.arange(b) % 7
        out = G.outage_deltas(g, yb, br)
    if form == "zip":
        rng = np.random.default_rng(n)
        z = 0.01 * (rng.random(n) + 1j * rng.random(n))
        topo.set_zip(z, z[::-1].copy())
    shared = topo.solve(p, q, vm, va, precision=prec, outage=out, history=True)
    rows = topo.solve(p, q, np.tile(vm, (b, 1)), np.tile(va, (b, 1)), precision=prec, outage=out,
                      history=True)
    for k in ("voltage_mag", "voltage_ang", "iterations", "status", "max_mismatch", "history"):
        np.testing.assert_array_equal(getattr(shared, k), getattr(rows, k), err_msg=k)
