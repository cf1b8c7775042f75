"""GPU: the solo programs (32 sums per warp, for batches of few scenarios).

A topology builds them with its tuning, or at its second solve of few scenarios;
they run the sums of the stream plans in the same order, so the solves must
equal the streams' results bit for bit: grids of a few buses and up to those with several CTAs per
scenario, one scenario, one more than a group, and as many as still run them.
On a small grid fewer launches than the first solve's show that the loop ran
in one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,batches", [(3, (1, 33)), (9, (2, 150)), (119, (1, 33, 600)), (700, (1, 33)),
                                       (2003, (1, 9)), (5003, (1,))])
def test_solo_equals_streams(n, batches, precision):
    import gridoxide_gb300 as gox
    from gridoxide_gb300 import grids as G
    from gridoxide_gb300 import solver as S

    prec = gox.GOX_PRECISION_MIXED if precision == "mixed" else gox.GOX_PRECISION_FP64
    g = G.family_grid(n, 3)
    yb = G.build_ybus(g)
    loads = {b: G.load_scenarios(g, b, 0.15, b) for b in batches}
    try:
        S.set_autotune(False)
        streams = gox.Topology(yb, g.bus_type)
        assert streams.prepare(g.p_spec, g.q_spec, g.vm, g.va)
        ref = {b: streams.solve(*loads[b], g.vm, g.va, precision=prec) for b in batches}
    finally:
        S.set_autotune(True)
    topo = gox.Topology(yb, g.bus_type)
    assert topo.prepare(g.p_spec, g.q_spec, g.vm, g.va)
    first = topo.solve(*loads[batches[0]], g.vm, g.va, precision=prec)
    launches = topo.last_launches()
    for b in batches:
        for _ in range(2):
            r = topo.solve(*loads[b], g.vm, g.va, precision=prec)
        if b == batches[0] and topo.tuning(prec)["chunk_words"] == 128 and n == 119:
            assert topo.last_launches() < launches  # the whole loop in one
        for k in ("voltage_mag", "voltage_ang", "iterations", "status", "max_mismatch"):
            np.testing.assert_array_equal(getattr(ref[b], k), getattr(r, k), err_msg=f"{n} {b} {k}")
    np.testing.assert_array_equal(first.voltage_mag, ref[batches[0]].voltage_mag)
