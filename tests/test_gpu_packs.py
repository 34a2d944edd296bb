"""The DP by packs of nets where it can go wrong, against the oracle.

Batch by batch the routes equal the oracle's DP on the GPU's own tables, and
the persistent executor (packs of several nets per warp when a batch has more
nets than warps) gives the same routes: every layer count's unrolled and
generic form including the ten layers whose arena holds fewer than 16 nodes;
capacities so small that via costs span many orders of magnitude (corner
columns whose sums round are added term by term); a batch larger than the GPU's
warps; a handful of nets; nets of one node and of none.
"""
import numpy as np
import pytest

import oracle
from helpers import orc_grid

pytestmark = pytest.mark.gpu

CASES = {
    "rough_24x24x10": dict(X=24, Y=24, cap_layers=10, n=1500, cap_lo=0, cap_hi=1, blockage=0.2, unit_via=1e-3),
    "tight_30x20x7": dict(X=30, Y=20, cap_layers=7, n=900, cap_lo=0, cap_hi=2, blockage=0.1, unit_via=0.5),
    "layers10_40x44x11": dict(X=40, Y=44, cap_layers=11, n=1200, cap_lo=1, cap_hi=4, max_pins=64, two_pin_frac=0.3),
    "layers3_33x50x4": dict(X=33, Y=50, cap_layers=4, n=700, cap_lo=1, cap_hi=4),
    "wide_batch_420x400x10": dict(X=420, Y=400, cap_layers=10, n=30000, cap_lo=4, cap_hi=9, bbox_median=2.5,
                                  two_pin_frac=0.6),
    "few_nets": dict(X=64, Y=64, cap_layers=10, n=3, cap_lo=1, cap_hi=3),
}


@pytest.mark.parametrize("case", list(CASES))
def test_packs_equal_oracle(case):
    from grotor_b200 import Router
    from grotor_b200.router import NetArrays
    from grotor_b200.synth import WORKLOADS, Design
    kw = dict(CASES[case])
    d = Design(WORKLOADS["small_64x64x5"].scaled(kw.pop("n"), seed=77, **kw))
    g, n = d.grid, d.nets
    # One net of a single node and one without nodes behind the design's.
    last = [np.append(a, [a[-1] + k, a[-1] + k]) for a, k in ((n.node_off, 1), (n.route_off, 9), (n.point_off, 0),
                                                              (n.hseg_off, 0), (n.vseg_off, 0))]
    nets = NetArrays(last[0], np.append(n.nodes, 0), np.append(n.parents, -1), last[1], last[2], n.points, last[3],
                     n.hsegs, last[4], n.vsegs)
    order = np.concatenate([d.order, [n.n, n.n + 1]]).astype(np.int32)
    og = orc_grid(g)
    with Router(g) as r:
        r.upload_nets(nets)
        _, nb = r.generate_batches_rsmt(order, 1000000)
        ids, off = r.plan()
        if case.startswith("wide"):
            assert np.diff(off).max() > 148 * 16
        rough = 0
        for b in range(nb):
            r.refresh_cost()
            t = r.read_tables()
            v = t["vcost"]
            rough += int(v.max() > 2.0 ** 26 * v.min())
            r.route_batch(b, b + 1)
            mine = r.read_routes()
            want = np.zeros_like(mine)
            sel = ids[off[b]:off[b + 1]]
            full = np.array([i for i in sel if nets.node_off[i + 1] > nets.node_off[i]], np.int32)
            assert oracle.lshape_batch(og, v, t["presum"], full, nets.node_off, nets.nodes, nets.parents,
                                       nets.route_off, want) == 0
            for i in full:
                a = nets.route_off[i]
                np.testing.assert_array_equal(mine[a:a + want[a]], want[a:a + want[a]], err_msg=f"net {i}, batch {b}")
            r.commit_batch_demand(b, b + 1, 1)
        if case.startswith("rough"):
            assert rough, "no via costs far apart"
        routes, dem, st = r.read_routes(), r.read_tables()["demand_half"], r.stats()
        r.reset()
        sp = r.lshape_route("persistent")
        np.testing.assert_array_equal(r.read_routes(), routes)
        np.testing.assert_array_equal(r.read_tables()["demand_half"], dem)
        assert sp["wirelength"] == st["wirelength"] and sp["vias"] == st["vias"]


@pytest.mark.parametrize("cap_layers", [10, 6, 11])
def test_trees_beyond_a_pack_equal_oracle(cap_layers):
    """Trees of 17 to 32 nodes (packs in global scratch) and of more (the general
    form, unrolled for nine layers), per batch and persistent."""
    from grotor_b200 import Router
    from grotor_b200.synth import WORKLOADS, Design
    d = Design(WORKLOADS["small_64x64x5"].scaled(160, seed=79, X=60, Y=52, cap_layers=cap_layers, cap_lo=1, cap_hi=4,
                                                max_pins=64, two_pin_frac=0.2, geo_p=0.05, bbox_median=25.0),
               max_subnet_pins=64)
    g, m = d.grid, d.nets
    sizes = np.diff(m.node_off)
    assert ((sizes > 16) & (sizes <= 32)).sum() > 10 and (sizes > 32).sum() > 10
    with Router(g) as r:
        r.upload_nets(m)
        _, nb = r.generate_batches_rsmt(d.order, 1000000)
        ids, off = r.plan()
        for b in range(nb):
            r.refresh_cost()
            t = r.read_tables()
            r.route_batch(b, b + 1)
            mine, want = r.read_routes(), np.zeros(int(m.route_off[-1]), np.int32)
            assert oracle.lshape_batch(orc_grid(g), t["vcost"], t["presum"], ids[off[b]:off[b + 1]], m.node_off, m.nodes,
                                       m.parents, m.route_off, want) == 0
            for i in ids[off[b]:off[b + 1]]:
                a = m.route_off[i]
                np.testing.assert_array_equal(mine[a:a + want[a]], want[a:a + want[a]], err_msg=f"net {i}, batch {b}")
            r.commit_batch_demand(b, b + 1, 1)
        routes, dem = r.read_routes(), r.read_tables()["demand_half"]
        r.reset()
        r.lshape_route("persistent")
        np.testing.assert_array_equal(r.read_routes(), routes)
        np.testing.assert_array_equal(r.read_tables()["demand_half"], dem)
