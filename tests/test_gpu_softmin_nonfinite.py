"""Soft-min inputs that are not finite.  A candidate whose cost is NaN, infinite
or at least 1e21 does not exist, whatever the size of its net: edges of infinite
and of NaN unit wire cost (every run over or behind one on its track drops out)
and an infinite via cost (only single-layer ranges are left).  A temperature whose
reciprocal is infinite is the hard minimum.  In fp64 against
the dense reference with such candidates dropped from every minimum; 1e-9 on the
cost and 1e-7 on the gradients as for finite inputs."""
import numpy as np
import pytest
import torch

import softmin_reference as R

pytestmark = pytest.mark.gpu


def _smin_of_existing(vals, tau):
    v = [x for x in vals if x is not None and bool(x < 1e21)]
    return -tau * torch.logsumexp(-torch.stack(v) / tau, dim=0) if v else None


def _design(kind):
    from grotor_b200.synth import WORKLOADS, Design
    if kind == "packs":
        return Design(WORKLOADS["small_64x64x5"].scaled(60, seed=81, X=20, Y=27, cap_layers=8))
    return Design(WORKLOADS["small_64x64x5"].scaled(14, seed=82, X=40, Y=36, cap_layers=6, max_pins=64, two_pin_frac=0.05,
                                                   geo_p=0.04, bbox_median=30.0), max_subnet_pins=64)


def _inputs(d, case, dtype=np.float64):
    g = d.grid
    rng = np.random.default_rng(9)
    uw = rng.uniform(0.5, 1.5, g.cells)
    at = rng.choice(g.cells, g.cells // 60, replace=False)
    uv = 1.5
    if case == "infinite_edges":
        uw[at] = np.inf
    elif case == "nan_edges":
        uw[at] = np.nan
    elif case == "huge_edges":  # finite, but no candidate: nothing lies behind them
        line = np.zeros((g.L, g.X, g.Y), bool)
        for l in range(g.L):
            if ((l & 1) ^ g.DIR) == 1:
                line[l, :, g.Y - 2] = rng.random(g.X) < 0.3
            else:
                line[l, g.X - 2, :] = rng.random(g.Y) < 0.3
        uw[line.reshape(-1)] = 1e25
    else:
        uv = np.inf
    return [torch.tensor(np.asarray(v, dtype), requires_grad=True) for v in (g.capacity.reshape(-1), uw, uv)]


@pytest.mark.parametrize("kind", ["packs", "big_trees"])
@pytest.mark.parametrize("case", ["infinite_edges", "nan_edges", "huge_edges", "infinite_vias"])
def test_candidates_that_do_not_exist(kind, case, monkeypatch):
    from grotor_b200 import Router
    from grotor_b200.softmin import routing_cost
    d = _design(kind)
    monkeypatch.setattr(R, "_smin", _smin_of_existing)
    p = _inputs(d, case)
    dem = np.zeros(d.grid.cells, np.int32)
    _, vc, P = R.tables(d.grid, dem, *p)
    m, tau = d.nets, 0.2
    costs = [R.net_cost(d.grid, vc, P, m.nodes[a:b], m.parents[a:b], tau) for a, b in zip(m.node_off[:-1], m.node_off[1:])]
    left = [c for c in costs if c is not None]
    total = sum(left, torch.zeros((), dtype=torch.float64, requires_grad=True))
    assert left or (kind, case) == ("big_trees", "infinite_vias")
    want = torch.autograd.grad(total, p, allow_unused=True, materialize_grads=True)
    q = [v.detach().cuda().requires_grad_(True) for v in p]
    with Router(d.grid) as r:
        r.upload_nets(m)
        F = routing_cost(r, *q, tau)
        got = torch.autograd.grad(F, q)
    # A net without a route counts 1e22 each.
    lost = len(costs) - len(left)
    assert F.item() == pytest.approx(total.item() + 1e22 * lost, rel=1e-9)
    for a, b in zip(got, want):
        assert bool(torch.isfinite(a).all())
        torch.testing.assert_close(a.cpu(), b.reshape(a.shape), rtol=1e-7, atol=1e-7 * float(b.abs().max()) + 1e-12)


@pytest.mark.parametrize("dtype,tau", [(torch.float32, 1e-40), (torch.float64, 1e-310)])
def test_temperature_below_the_reciprocal(dtype, tau):
    """Below any difference of two costs of the working precision the soft minimum
    is the hard one (ties apart: their count's logarithm is times tau)."""
    from grotor_b200 import Router
    from grotor_b200.softmin import routing_cost
    d = _design("packs")
    g = d.grid
    rng = np.random.default_rng(10)
    p = [torch.tensor(np.asarray(v, np.float64)) for v in (g.capacity.reshape(-1), rng.uniform(0.5, 1.5, g.cells), 2.0)]
    want = R.total_cost(g, np.zeros(g.cells, np.int32), d.nets, *p, 0).item()
    q = [v.to(dtype).cuda().requires_grad_(True) for v in p]
    with Router(g) as r:
        r.upload_nets(d.nets)
        F = routing_cost(r, *q, tau)
        got = torch.autograd.grad(F, q)
    assert F.item() == pytest.approx(want, rel=1e-5 if dtype == torch.float32 else 1e-12)
    assert all(bool(torch.isfinite(v).all()) for v in got)
