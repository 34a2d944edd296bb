"""The packed soft-min DP and adjoint where they can go wrong, in fp64 against
the dense PyTorch reference (1e-9 on the cost, 1e-7 on the gradients: sums of
a few thousand fp64 terms whose exponents' arguments are divided by tau):
trees that fit a pack, trees of 17 to 32 nodes, larger ones (walked by a
thread), several layer counts, nets of one node, and a design whose blocked
cells and full edges push candidates far apart.  Route transfers around a
soft-min call keep working (its workspace is its own)."""
import numpy as np
import pytest
import torch

import softmin_reference as R

pytestmark = pytest.mark.gpu

CASES = {
    "layers9": (dict(X=20, Y=27, cap_layers=10, max_pins=12), 70, 12, 0.1),
    "layers4_small_tau": (dict(X=33, Y=18, cap_layers=5, max_pins=12), 60, 12, 0.02),
    "layers2": (dict(X=12, Y=40, cap_layers=3, max_pins=8), 40, 8, 1.0),
    "layers10": (dict(X=16, Y=16, cap_layers=11, max_pins=12), 40, 12, 0.5),
    "big_trees": (dict(X=48, Y=44, cap_layers=7, max_pins=64, two_pin_frac=0.05, geo_p=0.04, bbox_median=30.0), 24, 64, 0.3),
    "blocked": (dict(X=20, Y=20, cap_layers=10, cap_lo=0, cap_hi=1, blockage=0.3), 50, 12, 0.1),
}


@pytest.mark.parametrize("case", list(CASES))
def test_packs_equal_dense_reference(case):
    from grotor_b200 import Router
    from grotor_b200.router import NetArrays
    from grotor_b200.softmin import routing_cost
    from grotor_b200.synth import WORKLOADS, Design
    kw, n, pins, tau = CASES[case]
    d = Design(WORKLOADS["small_64x64x5"].scaled(n, seed=31, **kw), max_subnet_pins=pins)
    g, m = d.grid, d.nets
    sizes = np.diff(m.node_off)
    if case == "big_trees":
        assert ((sizes > 16) & (sizes <= 32)).any() and (sizes > 32).any()
    nets = NetArrays(np.append(m.node_off, m.node_off[-1] + 1), np.append(m.nodes, 5), np.append(m.parents, -1),
                     np.append(m.route_off, m.route_off[-1] + 9), np.append(m.point_off, m.point_off[-1]), m.points,
                     np.append(m.hseg_off, m.hseg_off[-1]), m.hsegs, np.append(m.vseg_off, m.vseg_off[-1]), m.vsegs)
    cells = g.L * g.X * g.Y
    rng = np.random.default_rng(3)
    with Router(g) as r:
        r.upload_nets(nets)
        r.generate_batches_rsmt(np.append(d.order, m.n).astype(np.int32))
        r.lshape_route()
        dem = r.read_tables()["demand_half"]
        sent = r.read_routes_used(np.zeros(int(nets.route_off[-1]), np.int32))
        uw = g.unit_wire * rng.uniform(0.5, 1.5, cells)
        t = [torch.tensor(np.asarray(v, np.float64), device="cuda", requires_grad=True)
             for v in (g.capacity.reshape(-1), uw, g.unit_via)]
        F = routing_cost(r, *t, tau)
        got = torch.autograd.grad(F, t)
        np.testing.assert_array_equal(r.read_routes_used(np.zeros_like(sent)), sent)
        q = [v.detach().cpu().clone().requires_grad_(True) for v in t]
        W = R.total_cost(g, dem, nets, *q, tau)
        want = torch.autograd.grad(W, q)
        assert F.item() == pytest.approx(W.item(), rel=1e-9)
        for a, b in zip(got, want):
            torch.testing.assert_close(a.cpu(), b.reshape(a.shape), rtol=1e-7, atol=1e-7 * float(b.abs().max()))


CASES_F32 = {
    "layers9": (dict(X=20, Y=27, cap_layers=10, max_pins=12), 70, 12, 0.1),
    "layers10": (dict(X=16, Y=16, cap_layers=11, max_pins=12), 40, 12, 0.5),
    "layers4_small_tau": (dict(X=33, Y=18, cap_layers=5, max_pins=12), 60, 12, 0.05),
    "big_trees": (dict(X=48, Y=44, cap_layers=7, max_pins=64, two_pin_frac=0.05, geo_p=0.04, bbox_median=30.0), 24, 64, 4.0),
    "long_tracks": (dict(X=320, Y=18, cap_layers=6, max_pins=12, bbox_median=20.0), 60, 12, 0.5),
}


@pytest.mark.parametrize("case", list(CASES_F32))
def test_packs_in_fp32_agree_with_fp64(case):
    """The same inputs in both precisions.  A candidate's cost is off by at most
    delta: two prefix values rounded once each, and up to four roundings per tree
    node of a sum no larger than the net's cost.  So a cost is off by delta per
    net, a softmin weight by a factor exp(2 delta / tau) (numerator and sum), and
    an adjoint, a product of two weights (range and candidate) per level, by that
    factor to twice the depth; the cost model's own derivatives by a few times
    1e-6 (differences of exponentials of half a unit)."""
    from grotor_b200 import Router
    from grotor_b200.softmin import routing_cost
    from grotor_b200.synth import WORKLOADS, Design
    kw, n, pins, tau = CASES_F32[case]
    d = Design(WORKLOADS["small_64x64x5"].scaled(n, seed=32, **kw), max_subnet_pins=pins)
    g, m = d.grid, d.nets
    depth, dep = 0, np.zeros(len(m.nodes), np.int64)
    for a, b in zip(m.node_off[:-1], m.node_off[1:]):
        for k in range(a + 1, b):
            dep[k] = dep[a + m.parents[k]] + 1
    depth = int(dep.max())
    uw = np.random.default_rng(4).uniform(0.5, 1.5, g.cells).astype(np.float32)
    p = [np.asarray(g.capacity.reshape(-1), np.float32), uw, np.float32(g.unit_via)]
    out = {}
    with Router(g) as r:
        r.upload_nets(m)
        for dtype in (torch.float64, torch.float32):
            t = [torch.tensor(v, dtype=dtype, device="cuda", requires_grad=True) for v in p]
            F = routing_cost(r, *t, tau)
            out[dtype] = (F.item(), [v.double().cpu() for v in torch.autograd.grad(F, t)])
    _, vc, P = R.tables(g, np.zeros(g.cells, np.int32), *(torch.tensor(v, dtype=torch.float64) for v in p))
    nodes = int(np.diff(m.node_off).max())
    most = max(float(R.net_cost(g, vc, P, m.nodes[a:b], m.parents[a:b], tau)) for a, b in zip(m.node_off[:-1], m.node_off[1:]))
    delta = (2 * float(P.max()) + 4 * nodes * most) * 2.0 ** -24
    bound = np.expm1(4 * depth * delta / tau) + 1e-5
    assert bound < 0.4
    (f, want), (f32, got) = out[torch.float64], out[torch.float32]
    assert abs(f32 - f) <= m.n * delta + 1e-6 * abs(f)
    errors = [float((a - b).abs().max() / b.abs().max()) for a, b in zip(got, want)]
    assert max(errors) <= bound, (errors, bound)
