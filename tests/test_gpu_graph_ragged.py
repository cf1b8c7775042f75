"""GPU: ragged batches share the captured Newton loop of their group count.

A captured loop depends on the number of groups of 32 scenarios, not on how
many lanes of the last one are used: after a batch's second solve has captured
it, another scenario count of the same groups runs it at its first solve, with
the results of a topology that never captures, bit for bit."""
import numpy as np
import pytest

from gridoxide_gb300 import grids as G
from helpers import grid_from_fixture, load_fixture, ybus_from_fixture

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_ragged_batches_share_the_captured_loop(gox, precision):
    prec = gox.GOX_PRECISION_MIXED if precision == "mixed" else gox.GOX_PRECISION_FP64
    fx = load_fixture("case118")
    g, yb = grid_from_fixture(fx), ybus_from_fixture(fx)
    p, q = G.load_scenarios(g, 2080, 0.15, 43)  # 65 groups: 2,049 to 2,080 scenarios
    topo, host = gox.Topology(yb, g.bus_type), gox.Topology(yb, g.bus_type)
    host.set_graph(False)
    solve = lambda t, b: t.solve(p[:b], q[:b], g.vm, g.va, precision=prec)  # noqa: E731
    for _ in range(2):
        solve(topo, 2080)
    ran = topo.info()["graph_solves"]
    assert ran == 1
    for b in (2049, 2063, 2079, 2080, 2050):
        r, ref = solve(topo, b), solve(host, b)
        ran += 1
        assert topo.info()["graph_solves"] == ran, b
        for k in ("voltage_mag", "voltage_ang", "iterations", "status", "max_mismatch"):
            np.testing.assert_array_equal(getattr(r, k), getattr(ref, k), err_msg=f"{b} {k}")
