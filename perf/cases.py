"""The power-flow work that users of this framework have it do, as cases to measure.

Each case is one call of a public entry point on a grid of the synthetic
meshed family (`gridoxide_gb300.grids`): the grid and its registered topology
are what a program keeps between calls, so they are built once per process;
the injections, start points and outages are new for every seed.

    listed()              the cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   inputs and handles, as a program has them before the call
    run(state)            one call, its whole result
    work(case)            the bytes and operations of one call
    exact(case, seed)     the solution in 64 bits by plain numpy / torch
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gridoxide_gb300 as gox
from gridoxide_gb300 import grids as G

TOL = 1e-8
PRECISION = {"mixed": gox.GOX_PRECISION_MIXED, "fp64": gox.GOX_PRECISION_FP64}
DENSE_UNKNOWNS = 4500  # exact() solves dense systems up to this size


def listed():
    return [
        # one power flow of a small grid from a flat start: the interactive
        # call, where launches and the dependency chain are all there is
        dict(name="single_118_fp64", kind="host", grid="case118", batch=1, precision="fp64",
             start="flat", outage=False),
        # one request of a serving loop: a mid-size grid, warm start, a branch
        # out
        dict(name="request_1500_mixed", kind="host", grid="family", n=1500, grid_seed=21, batch=1,
             precision="mixed", start="warm", outage=True),
        # one request on a large grid: most of its columns are in a few wide
        # levels, one group of scenarios
        dict(name="request_20000_mixed", kind="host", grid="family", n=20000, grid_seed=22, batch=1,
             precision="mixed", start="warm", outage=False),
        # a few load cases of a district grid with host arrays, ragged batch
        dict(name="loadcases_300x75_mixed", kind="host", grid="family", n=300, grid_seed=23,
             batch=75, precision="mixed", start="flat", outage=False),
        # a month of quarter-hour load profiles of a small grid, FP64, on
        # torch's current stream
        dict(name="profiles_118x2976_fp64", kind="device", grid="case118", batch=2976,
             precision="fp64", start="flat", outage=False, stream="current"),
        # Monte-Carlo load scenarios of a transmission grid: the batch the
        # benchmark quotes, inputs on the device, a stream of its own
        dict(name="batch_2000x4096_mixed", kind="device", grid="case2000", batch=4096,
             precision="mixed", start="flat", outage=False, stream="own"),
        # the same grid in plain FP64, a ragged batch
        dict(name="batch_2000x1500_fp64", kind="device", grid="case2000", batch=1500,
             precision="fp64", start="flat", outage=False, stream="own"),
        # a screening batch with host arrays: copies in and out are the call's
        dict(name="screen_2000x999_mixed", kind="host", grid="case2000", batch=999,
             precision="mixed", start="flat", outage=False),
        # N-1 contingency screen of a 10,000-bus grid, warm start from the
        # base case, one non-bridge branch out per scenario, on torch's current
        # stream
        dict(name="n1_10000x4096_mixed", kind="device", grid="case10000", batch=4096,
             precision="mixed", start="warm", outage=True, stream="current"),
        # uniform load scalings with the linear initial guess (the PGM batch
        # workflow), FP64
        dict(name="scaled_1000x512_fp64", kind="scaled", grid="family", n=1000, grid_seed=24,
             batch=512, precision="fp64"),
        # uneven batch over several topologies in one call
        dict(name="many_8_mixed", kind="many", count=8, n_min=30, n_max=3000, b_min=8, b_max=512,
             grid_seed=25, precision="mixed"),
        # the LinearSolver drop-in: one Newton step's refactor and solve from
        # host values
        dict(name="linear_2000_fp64", kind="linear", grid="case2000"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "device", "device", "n1", "scaled", "linear", "many"])
    gs = rng.randrange(100, 10000)
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "host":  # requests and small batches with host arrays
        n = _log(rng, 30, 12000)
        return dict(kind="host", grid="family", n=n, grid_seed=gs,
                    batch=1 if rng.random() < 0.5 else _log(rng, 1, max(2, min(999, 2000000 // n))),
                    precision=precision, start=rng.choice(["flat", "warm"]),
                    outage=rng.random() < 0.3)
    if kind == "device":
        n = _log(rng, 50, 4000)
        top = 8000000 if precision == "mixed" else 3000000
        return dict(kind="device", grid="family", n=n, grid_seed=gs,
                    batch=_log(rng, 32, min(8192, top // n)), precision=precision, start="flat",
                    outage=False, stream=rng.choice(["current", "own"]))
    if kind == "n1":
        n = _log(rng, 500, 10000)
        return dict(kind="device", grid="family", n=n, grid_seed=gs,
                    batch=_log(rng, 64, min(4096, 20000000 // n)), precision="mixed", start="warm",
                    outage=True, stream=rng.choice(["current", "own"]))
    if kind == "scaled":
        n = _log(rng, 50, 2500)
        return dict(kind="scaled", grid="family", n=n, grid_seed=gs,
                    batch=_log(rng, 8, min(2048, 1000000 // n)), precision=precision)
    if kind == "many":
        return dict(kind="many", count=rng.randrange(3, 8), n_min=30, n_max=_log(rng, 300, 3000),
                    b_min=8, b_max=_log(rng, 16, 512), grid_seed=gs, precision=precision)
    return dict(kind="linear", grid="family", n=_log(rng, 30, 2200), grid_seed=gs)


# ---------------------------------------------------------------------------
# Grids and handles: one per process and grid, as a program keeps them

class _Net:
    """A grid, its Y-bus and (on first use) its registered topology with the
    base case's pivot order and voltages."""

    def __init__(self, grid):
        self.g = grid
        self.yb = G.build_ybus(grid)
        self._topo = None
        self._warm = None
        self._safe = None
        self._solver = None

    @property
    def topo(self):
        if self._topo is None:
            self._topo = gox.Topology(self.yb, self.g.bus_type)
            # the pivot order comes from the base case, whatever batch is
            # solved first
            self._topo.prepare(self.g.p_spec, self.g.q_spec, self.g.vm, self.g.va, tol=TOL)
        return self._topo

    def warm(self):
        """The base case's voltages."""
        if self._warm is None:
            r = self.topo.solve(self.g.p_spec, self.g.q_spec, self.g.vm, self.g.va, tol=TOL,
                                precision=gox.GOX_PRECISION_FP64)
            self._warm = (r.voltage_mag[0].copy(), r.voltage_ang[0].copy())
        return self._warm

    def safe_branches(self):
        """The branches whose loss leaves the grid in one piece."""
        if self._safe is None:
            self._safe = np.flatnonzero(~G.bridges(self.g))
        return self._safe

    def solver(self):
        """(rows, cols, LinearSolver) of the Jacobian pattern at the base case."""
        if self._solver is None:
            jac = _Jacobian(self.g, self.yb)
            vals = jac.values(self.g.vm, self.g.va)
            entries = list(zip(jac.rows.tolist(), jac.cols.tolist(), vals.tolist()))
            self._solver = (jac, gox.Gb300LinearSolver.new(jac.n_u, entries))
        return self._solver


_NETS: dict = {}


def _net(case, n=None, seed=None):
    key = (case.get("grid", "family"), n if n is not None else case.get("n"),
           seed if seed is not None else case.get("grid_seed"))
    if key not in _NETS:
        _NETS[key] = _Net(G.config_grid(key[0]) if key[0] != "family"
                          else G.family_grid(key[1], key[2]))
    return _NETS[key]


def _many(case):
    """[(net, batch)] of a many-topology case."""
    rng = np.random.default_rng(case["grid_seed"])
    ns = np.exp(rng.uniform(np.log(case["n_min"]), np.log(case["n_max"]), case["count"])).astype(int)
    bs = rng.integers(case["b_min"], case["b_max"] + 1, case["count"])
    return [(_net({"grid": "family"}, int(n), 1000 + case["grid_seed"] + k), int(b))
            for k, (n, b) in enumerate(zip(ns, bs))]


# ---------------------------------------------------------------------------
# Inputs

def _outages(net, batch, seed):
    pick = np.random.default_rng(seed).choice(net.safe_branches(), batch)
    return G.outage_deltas(net.g, net.yb, pick)


def _loads(net, batch, seed):
    """[batch, n] injections on the GPU: every load x lognormal(0, 0.15), the
    generation rescaled to the scenario's load."""
    g = net.g
    gen = torch.Generator(device="cuda").manual_seed(seed)
    mult = torch.randn(batch, g.n_bus, generator=gen, device="cuda", dtype=torch.float64).mul_(0.15).exp_()
    share = torch.tensor(1.03 * g.pv_weight / g.pv_weight.sum(), device="cuda")
    p = mult * torch.tensor(g.load_p, device="cuda")
    p = p.sum(1, keepdim=True) * share - p
    q = mult * torch.tensor(-g.load_q, device="cuda")
    return p, q


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind)
    if kind == "linear":
        net = _net(case)
        jac, solver = net.solver()
        rng = np.random.default_rng(seed)
        n = net.g.n_bus
        vm = net.g.vm * rng.uniform(0.98, 1.02, n)
        va = rng.uniform(-0.05, 0.05, n)
        s.update(solver=solver, values=jac.values(vm, va), rhs=rng.normal(0.0, 0.05, jac.n_u))
        return s
    s["precision"] = PRECISION[case["precision"]]
    if kind == "many":
        jobs = []
        for k, (net, b) in enumerate(_many(case)):
            p, q = _loads(net, b, seed * 64 + k)
            jobs.append((net.topo, p.cpu().numpy(), q.cpu().numpy(), net.g.vm, net.g.va))
        s["jobs"] = jobs
        return s
    net = _net(case)
    b, n = case["batch"], net.g.n_bus
    s["topo"] = net.topo
    if kind == "scaled":
        s["scales"] = np.random.default_rng(seed).uniform(0.8, 1.2, b)
        s["base"] = (net.g.p_spec, net.g.q_spec, net.g.vm, net.g.va)
        return s
    p, q = _loads(net, b, seed)
    vm, va = net.warm() if case["start"] == "warm" else (net.g.vm, net.g.va)
    outage = _outages(net, b, seed) if case["outage"] else None
    if kind == "host":
        s.update(p=p.cpu().numpy(), q=q.cpu().numpy(), vm=vm, va=va, outage=outage)
        return s
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    new = lambda shape, dt: torch.empty(shape, dtype=dt, device="cuda")  # noqa: E731
    s.update(p=p, q=q, vm=dev(vm), va=dev(va),
             outage=tuple(dev(a) for a in outage) if outage is not None else None,
             out=(new((b, n), torch.float64), new((b, n), torch.float64), new((b,), torch.int32),
                  new((b,), torch.int32), new((b,), torch.float64)))
    s["stream"] = torch.cuda.Stream() if case["stream"] == "own" else torch.cuda.current_stream()
    s["stream"].wait_stream(torch.cuda.current_stream())  # the inputs above
    return s


# ---------------------------------------------------------------------------
# The calls

def run(s):
    kind = s["kind"]
    if kind == "linear":
        return s["solver"].factor_and_solve_values(s["values"], s["rhs"])
    if kind == "many":
        return [_fields(r) for r in gox.multi_solve(s["jobs"], tol=TOL, precision=s["precision"])]
    topo = s["topo"]
    if kind == "scaled":
        topo.set_initial_guess("linear")
        try:
            return _fields(topo.solve_scaled(s["scales"], *s["base"], tol=TOL, precision=s["precision"]))
        finally:
            topo.set_initial_guess("given")
    if kind == "host":
        return _fields(topo.solve(s["p"], s["q"], s["vm"], s["va"], tol=TOL,
                                  precision=s["precision"], outage=s["outage"]))
    topo.solve_device(s["p"], s["q"], s["vm"], s["va"], *s["out"], tol=TOL,
                      precision=s["precision"], outage=s["outage"],
                      stream=s["stream"])
    vm, va, it, st, mm = s["out"]
    return dict(vm=vm, va=va, iterations=it, status=st, max_mismatch=mm)


def _fields(r):
    return dict(vm=r.voltage_mag, va=r.voltage_ang, iterations=r.iterations, status=r.status,
                max_mismatch=r.max_mismatch)


# ---------------------------------------------------------------------------
# What a call cannot do without

ITERATIONS = 5  # Newton steps of a converging solve


def _solve_work(n, batch, steps):
    # per bus: 3.8 Y entries (8 operations each, 16 bytes), a refactor of
    # about 120 operations and substitutions of about 85
    return dict(bytes=32.0 * batch * n + 16.0 * 3.8 * n,
                flops=float(steps) * batch * n * (120 + 85 + 40))


def work(case):
    kind = case["kind"]
    if kind == "many":
        rng = np.random.default_rng(case["grid_seed"])
        ns = np.exp(rng.uniform(np.log(case["n_min"]), np.log(case["n_max"]), case["count"])).astype(int)
        bs = rng.integers(case["b_min"], case["b_max"] + 1, case["count"])
        parts = [_solve_work(int(n), int(b), ITERATIONS) for n, b in zip(ns, bs)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["n"] if case["grid"] == "family" else G.CONFIGS[case["grid"]][0]
    if kind == "linear":  # 13 Jacobian entries per bus, the right-hand side, the solution
        return dict(bytes=8.0 * n * (13 + 2 * 1.85), flops=float(n) * (120 + 85))
    w = _solve_work(n, case["batch"], ITERATIONS)
    if kind == "scaled":  # the injections are expanded from one row
        w["bytes"] = 16.0 * case["batch"] * n + 32.0 * n
    return w


# ---------------------------------------------------------------------------
# The same solutions in 64 bits, from the equations alone

class _Jacobian:
    """Polar power-flow Jacobian of [P(non-slack); Q(PQ)] by [theta; |V|], as
    triplets over the Y-bus pattern."""

    def __init__(self, g, yb):
        n = g.n_bus
        self.i = np.repeat(np.arange(n), np.diff(yb.indptr))
        self.k = yb.indices.astype(np.int64)
        self.y = yb.re + 1j * yb.im
        self.ns = np.flatnonzero(g.bus_type != G.BUS_SLACK)
        self.pq = np.flatnonzero(g.bus_type == G.BUS_PQ)
        self.n_u = self.ns.size + self.pq.size
        at_a = np.full(n, -1)
        at_a[self.ns] = np.arange(self.ns.size)
        at_v = np.full(n, -1)
        at_v[self.pq] = self.ns.size + np.arange(self.pq.size)
        self.parts = []  # (entries of the Y pattern, rows, columns) of H, N, M, L
        for r, c in ((at_a, at_a), (at_a, at_v), (at_v, at_a), (at_v, at_v)):
            e = np.flatnonzero((r[self.i] >= 0) & (c[self.k] >= 0))
            self.parts.append((e, r[self.i[e]], c[self.k[e]]))
        self.rows = np.concatenate([p[1] for p in self.parts]).astype(np.int32)
        self.cols = np.concatenate([p[2] for p in self.parts]).astype(np.int32)
        self.diag = self.i == self.k

    def values(self, vm, va, y=None):
        y = self.y if y is None else y
        v = vm * np.exp(1j * va)
        cur = np.zeros(vm.size, complex)
        np.add.at(cur, self.i, y * v[self.k])
        s = v * np.conj(cur)
        t = v[self.i] * np.conj(y * v[self.k])  # the entry's share of S_i
        d_a = np.where(self.diag, 1j * (s[self.i] - t), -1j * t)
        d_v = t / vm[self.k] + np.where(self.diag, s[self.i] / vm[self.i], 0.0)
        full = (d_a.real, d_v.real, d_a.imag, d_v.imag)
        return np.concatenate([f[p[0]] for f, p in zip(full, self.parts)])

    def dense(self, vm, va, y=None):
        a = np.zeros((self.n_u, self.n_u))
        np.add.at(a, (self.rows, self.cols), self.values(vm, va, y))
        return a


def _newton_one(jac, p, q, vm, va, y):
    """Newton-Raphson of one scenario with dense solves, to the rounding floor."""
    vm, va = vm.copy(), va.copy()
    best = np.inf
    for _ in range(40):
        v = vm * np.exp(1j * va)
        cur = np.zeros(vm.size, complex)
        np.add.at(cur, jac.i, y * v[jac.k])
        s = v * np.conj(cur)
        f = np.concatenate([(p - s.real)[jac.ns], (q - s.imag)[jac.pq]])
        m = np.abs(f).max()
        if m < 1e-9 and m > 0.3 * best:
            break
        best = min(best, m)
        a = torch.from_numpy(jac.dense(vm, va, y)).cuda()
        dx = torch.linalg.solve(a, torch.from_numpy(f).cuda()).cpu().numpy()
        va[jac.ns] += dx[:jac.ns.size]
        vm[jac.pq] += dx[jac.ns.size:]
    return vm, va


def _newton_many(jac, p, q, vm0, va0):
    """[B, n] scenarios by Newton steps with the mean scenario's Jacobian."""
    b, n = p.shape
    mvm, mva = _newton_one(jac, p.mean(0).cpu().numpy(), q.mean(0).cpu().numpy(), vm0, va0, jac.y)
    lu = torch.linalg.lu_factor(torch.from_numpy(jac.dense(mvm, mva)).cuda())
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    i, k, y, ns, pq = dev(jac.i), dev(jac.k), dev(jac.y), dev(jac.ns), dev(jac.pq)
    vm, va = dev(mvm)[:, None].repeat(1, b), dev(mva)[:, None].repeat(1, b)
    pt, qt = p.T.contiguous(), q.T.contiguous()
    best = math.inf
    for _ in range(80):
        v = torch.polar(vm, va)
        cur = torch.zeros(n, b, dtype=torch.complex128, device="cuda")
        cur.index_add_(0, i, y[:, None] * v[k])
        s = v * cur.conj()
        f = torch.cat([(pt - s.real)[ns], (qt - s.imag)[pq]])
        m = float(f.abs().max())
        if not math.isfinite(m):
            return None
        if m < 1e-9 and m > 0.5 * best:
            break
        best = min(best, m)
        dx = torch.linalg.lu_solve(*lu, f)
        va[ns] += dx[:ns.numel()]
        vm[pq] += dx[ns.numel():]
    if best > 1e-9:
        return None
    return vm.T.contiguous(), va.T.contiguous()


def _exact_batch(net, p, q, vm0, va0, outage=None):
    none = dict(vm=None, va=None, iterations=None, status=None, max_mismatch=None)
    jac = _Jacobian(net.g, net.yb)
    if jac.n_u > DENSE_UNKNOWNS:
        return none
    if p.shape[0] <= 4:
        rows = []
        for r in range(p.shape[0]):
            y = jac.y.copy()
            if outage is not None:
                np.add.at(y, outage[0][r], outage[1][r] + 1j * outage[2][r])
            rows.append(_newton_one(jac, p[r].cpu().numpy(), q[r].cpu().numpy(), vm0, va0, y))
        return dict(none, vm=np.stack([r[0] for r in rows]), va=np.stack([r[1] for r in rows]))
    if outage is not None:  # every scenario has a Jacobian of its own
        return none
    got = _newton_many(jac, p, q, vm0, va0)
    return none if got is None else dict(none, vm=got[0], va=got[1])


def exact(case, seed):
    """What run() returns in 64 bits; None where no output has such a value."""
    got = _exact(case, seed)
    parts = got if isinstance(got, list) else [got]
    if all(isinstance(r, dict) and all(v is None for v in r.values()) for r in parts):
        return None
    return got


def _exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        net = _net(case)
        s = prepare(case, seed)
        jac = _Jacobian(net.g, net.yb)
        a = np.zeros((jac.n_u, jac.n_u))
        np.add.at(a, (jac.rows, jac.cols), s["values"])
        return torch.linalg.solve(torch.from_numpy(a).cuda(), torch.from_numpy(s["rhs"]).cuda())
    if kind == "many":
        return [_exact_batch(net, *_loads(net, b, seed * 64 + k), net.g.vm, net.g.va)
                for k, (net, b) in enumerate(_many(case))]
    net = _net(case)
    vm, va = net.g.vm, net.g.va
    if kind == "scaled":
        f = torch.from_numpy(np.random.default_rng(seed).uniform(0.8, 1.2, case["batch"])).cuda()
        p = f[:, None] * torch.from_numpy(net.g.p_spec).cuda()
        q = f[:, None] * torch.from_numpy(net.g.q_spec).cuda()
        return _exact_batch(net, p, q, vm, va)
    p, q = _loads(net, case["batch"], seed)
    return _exact_batch(net, p, q, vm, va, _outages(net, case["batch"], seed) if case["outage"] else None)
