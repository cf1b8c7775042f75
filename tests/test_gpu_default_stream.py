"""GPU: large device batches on the default stream run on a stream of their own,
after what the default stream holds and before what follows on it.

The inputs are written on the default stream right before the call, behind work
that takes a while, and the outputs are read on it right after; the result must
be that of a solve on a stream of its own, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,precision", [(2016, "mixed"), (2017, "mixed"), (2500, "fp64"), (4099, "mixed")])
def test_default_stream_order(b, precision):
    import torch
    import gridoxide_gb300 as gox
    from gridoxide_gb300 import grids as G

    prec = gox.GOX_PRECISION_MIXED if precision == "mixed" else gox.GOX_PRECISION_FP64
    n = 119
    g = G.family_grid(n, 3)
    yb = G.build_ybus(g)
    topo = gox.Topology(yb, g.bus_type)
    p, q = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in G.load_scenarios(g, b, 0.1, b))
    vm, va = torch.from_numpy(g.vm).cuda(), torch.from_numpy(g.va).cuda()

    def outputs():
        f = lambda s, d: torch.zeros(s, dtype=d, device="cuda")  # noqa: E731
        return (f((b, n), torch.float64), f((b, n), torch.float64), f((b,), torch.int32),
                f((b,), torch.int32), f((b,), torch.float64))

    own = torch.cuda.Stream()
    torch.cuda.synchronize()
    ref = outputs()
    for _ in range(3):
        topo.solve_device(p, q, vm, va, *ref, precision=prec, stream=own)
    torch.cuda.synchronize()
    assert bool((ref[3] == 0).all())
    big = torch.randn(4096, 4096, device="cuda")
    for _ in range(3):
        p2, q2, out = torch.full_like(p, float("nan")), torch.full_like(q, float("nan")), outputs()
        x = big
        for _ in range(8):
            x = x @ big * 1e-2
        p2.copy_(p)
        q2.copy_(q)
        topo.solve_device(p2, q2, vm, va, *out, precision=prec)
        copies = [t.clone() for t in out]
        for t in out:
            t.zero_()
        for a, c in zip(ref, copies):
            assert torch.equal(a, c)
