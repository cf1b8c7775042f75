"""GPU: what creating a linear solver costs.

It compiles the streams, a dot program and a solo program side by side, so it
takes little longer than registering and analysing the same pattern as a
topology, which compiles the streams only: one after the other they took 1.9
times that (2,003 buses; side by side 1.1)."""
import time

import numpy as np
import pytest

from gridoxide_gb300 import grids as G

pytestmark = pytest.mark.gpu


def test_linear_solver_creation(gox):
    from perf.cases import _Jacobian
    g = G.family_grid(2003, 3)
    yb = G.build_ybus(g)
    jac = _Jacobian(g, yb)
    values = jac.values(g.vm, g.va)
    entries = list(zip(jac.rows.tolist(), jac.cols.tolist(), values.tolist()))
    create, analyse = [], []
    for _ in range(6):
        t0 = time.perf_counter()
        solver = gox.Gb300LinearSolver.new(jac.n_u, entries)
        t1 = time.perf_counter()
        topo = gox.Topology(yb, g.bus_type)
        assert topo.prepare(g.p_spec, g.q_spec, g.vm, g.va)
        create.append(t1 - t0)
        analyse.append(time.perf_counter() - t1)
    assert min(create) <= 1.4 * min(analyse), (create, analyse)
    x = solver.factor_and_solve_values(values, np.ones(jac.n_u))
    r = np.bincount(jac.rows, values * x[jac.cols], jac.n_u) - 1.0
    assert np.abs(r).max() < 1e-8
