"""The Z-shape stage and the bounding-box rounds where their forms change,
against the oracle: nets whose arrays fit shared memory and nets of hundreds of
nodes whose arrays are in global scratch; edges shorter and longer than a
warp's chunk of positions; 3, 9 and 10 routable layers; nodes that share a position;
groups below, at and above the CTA's window with rounds of one net, of a few
and of as many as one may hold.
"""
import numpy as np
import pytest

import oracle
from helpers import orc_grid

pytestmark = pytest.mark.gpu

CASES = {
    "long_edges_200x18x10": dict(n=150, X=200, Y=18, cap_layers=10, pin_model=1, max_pins=256, pareto_alpha=0.7,
                                 bbox_model=1, bbox_max=200),
    "many_layers_40x44x11": dict(n=300, X=40, Y=44, cap_layers=11, max_pins=64, two_pin_frac=0.3),
    "few_layers_33x64x4": dict(n=300, X=33, Y=64, cap_layers=4, max_pins=64, two_pin_frac=0.3),
}


@pytest.mark.parametrize("case", list(CASES))
def test_zshape_equals_oracle(case):
    from grotor_b200 import Router
    from grotor_b200.router import NetArrays
    from grotor_b200.synth import WORKLOADS, Design
    kw = dict(CASES[case])
    d = Design(WORKLOADS["small_64x64x5"].scaled(kw.pop("n"), seed=61, cap_lo=1, cap_hi=4, **kw), max_subnet_pins=256)
    g, n, z = d.grid, d.nets, d.zshape_trees()
    zn = np.diff(z["node_off"]).astype(np.int64)
    if case.startswith("long"):
        assert zn.max() > 96 and zn.min() < 8
    route_off = np.concatenate([[0], np.cumsum(1 + 64 * zn)]).astype(np.int64)
    nets = NetArrays(n.node_off, n.nodes, n.parents, route_off, n.point_off, n.points, n.hseg_off, n.hsegs,
                     n.vseg_off, n.vsegs)
    og = orc_grid(g)
    og = oracle.OrcGrid(og.L, og.X, og.Y, og.DIR, og.unit_wire, og.unit_via, og.short_costs, og.x_edge_len,
                        og.y_edge_len, og.capacity, og.of_cost_scale, integer_wire=True)
    with Router(g) as r:
        r.upload_nets(nets)
        r.upload_zshape(z)
        r.set_wire_cost_mode(True)
        r.generate_batches_rsmt(d.order, 1000000)
        r.plan_bbox_batches(250)
        ids, off = r.plan()
        want = oracle.zshape_stage(og, z, ids, off, route_off)
        assert want["status"] == 0
        for mode in ("persistent", "plain"):
            r.reset()
            st = r.zshape_route(mode)
            np.testing.assert_array_equal(r.read_routes(), want["routes"])
            np.testing.assert_array_equal(r.read_tables()["demand_half"], want["demand_half"])
            assert st["wirelength"] == want["wirelength"] and st["vias"] == want["vias"]


@pytest.mark.parametrize("max_batch", [1, 7, 256])
def test_bbox_rounds_equal_oracle(max_batch):
    from grotor_b200 import Router
    from grotor_b200.synth import WORKLOADS, Design
    d = Design(WORKLOADS["small_64x64x5"].scaled(3500, seed=62))
    X, Y, n = d.grid.X, d.grid.Y, d.nets.n
    rng = np.random.default_rng(63)
    size = np.where(rng.random((n, 2)) < 0.8, rng.integers(1, 5, (n, 2)), rng.integers(1, 50, (n, 2)))
    at = (rng.random((n, 2)) * (np.array([X, Y]) - size + 1)).astype(np.int64)
    bbox = np.stack([at[:, 0], at[:, 0] + size[:, 0] - 1, at[:, 1], at[:, 1] + size[:, 1] - 1], 1).astype(np.int32)
    off = np.cumsum([0, 1, 31, 32, 255, 256, 257, 700, 1300])
    assert off[-1] <= n
    order = rng.permutation(n)[:off[-1]].astype(np.int32)
    want = []
    for k in range(len(off) - 1):  # groups in order, each one's rounds last first
        want += oracle.bbox_batches(X, Y, order[off[k]:off[k + 1]], bbox.reshape(-1), max_batch)[::-1]
    with Router(d.grid) as r:
        r.upload_nets(d.nets)
        r.upload_zshape(d.zshape_trees())
        r.set_plan(order, off.astype(np.int32))
        nb = r.plan_bbox_batches(max_batch, bbox)
        ids, got = r.plan()
        assert nb == len(want)
        np.testing.assert_array_equal(np.diff(got), [len(w) for w in want])
        np.testing.assert_array_equal(ids, np.concatenate(want))


@pytest.mark.parametrize("many", [False, True])
def test_scratch_follows_the_large_nets(many):
    """Nets of more than 96 nodes: a few of up to three hundred among small ones
    take memory for their own arrays, not for one such net on every block; where
    there are so many that a place per block is less, they share those."""
    import torch
    from grotor_b200 import Router
    from grotor_b200.router import NetArrays
    from grotor_b200.synth import WORKLOADS, Design
    if many:
        d = Design(WORKLOADS["small_64x64x5"].scaled(2400, seed=65, X=120, Y=120, cap_layers=4, two_pin_frac=0.0,
                                                    geo_p=0.001, max_pins=100, bbox_median=40.0, cap_lo=900, cap_hi=900), max_subnet_pins=256)
    else:
        d = Design(WORKLOADS["small_64x64x5"].scaled(400, seed=64, X=90, Y=90, cap_layers=10, pin_model=1, max_pins=256,
                                                    pareto_alpha=0.9, bbox_model=1, bbox_max=90), max_subnet_pins=256)
    n, z = d.nets, d.zshape_trees()
    zn = np.diff(z["node_off"]).astype(np.int64)
    wide, blocks = zn[zn > 96], 8 * torch.cuda.get_device_properties(0).multi_processor_count
    assert (wide.sum() > blocks * zn.max()) == many and len(wide)
    arrays = 4 * min(int(wide.sum()), int(blocks * zn.max())) * (18 * (d.grid.L + 1) + 10)
    room = np.concatenate([[0], np.cumsum(1 + 64 * zn)]).astype(np.int64)
    with Router(d.grid) as r:
        r.upload_nets(NetArrays(n.node_off, n.nodes, n.parents, room, n.point_off, n.points, n.hseg_off, n.hsegs,
                                n.vseg_off, n.vsegs))
        before = torch.cuda.mem_get_info()[0]
        r.upload_zshape(z)
        taken = before - torch.cuda.mem_get_info()[0]
        assert taken < arrays + (24 << 20), (taken, arrays)  # allocations come in 2 MiB pieces
        r.generate_batches_rsmt(d.order, 1000000)
        r.plan_bbox_batches(250)
        out = []
        for mode in ("persistent", "plain", "graph"):
            r.reset()
            r.zshape_route(mode)
            out.append(r.read_routes())
        np.testing.assert_array_equal(out[0], out[1])
        np.testing.assert_array_equal(out[0], out[2])
