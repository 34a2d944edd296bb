"""A plan and what is derived from it -- size buckets, captured stages -- stay
right when the context changes around them: scratch that another executor has
replaced by a larger one; other nets uploaded under the same plan; the other
wire-cost rule.  A fresh
context's plain executor, which keeps nothing, gives the expected routes."""
import numpy as np
import pytest

from helpers import flt_by_net, golden_grid, golden_nets, load_golden

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def big_nets():
    """Nets of 17 and more tree nodes, whose DP runs in global scratch, in
    batches of far fewer nets than the GPU has warps."""
    from grotor_b200.synth import WORKLOADS, Design
    d = Design(WORKLOADS["medium_320x320x10"].scaled(600, seed=45, two_pin_frac=0.2, geo_p=0.06, bbox_median=20.0),
               max_subnet_pins=64)
    sizes = np.diff(d.nets.node_off)
    assert ((sizes > 16) & (sizes <= 32)).any() and (sizes > 32).any()
    return d


def _stage(r, mode):
    r.reset()
    st = r.lshape_route(mode)
    return r.read_routes(), r.read_tables()["demand_half"], st["wirelength"], st["vias"]


def _same(got, want):
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
    assert got[2:] == want[2:]


def test_graph_after_the_scratch_grew(big_nets):
    """The graph captures the scratch of its largest batch; the persistent
    executor wants a slot per warp of the GPU and replaces it; the graph of the
    same plan then runs on the scratch that is there."""
    from grotor_b200 import Router
    d = big_nets
    with Router(d.grid) as r:
        r.upload_nets(d.nets)
        r.generate_batches_rsmt(d.order, 1000000)
        _, off = r.plan()
        assert np.diff(off).max() + 8 < 148 * 16
        want = _stage(r, "plain")
    with Router(d.grid) as r:
        r.upload_nets(d.nets)
        r.generate_batches_rsmt(d.order, 1000000)
        for mode in ("graph", "persistent", "graph", "plain", "graph"):
            _same(_stage(r, mode), want)


@pytest.mark.parametrize("mode", ["plain", "graph", "persistent"])
def test_plan_kept_over_an_upload_of_other_nets(big_nets, mode):
    """The same ids under the same plan, first with two-pin trees and then with
    trees of up to dozens of nodes (other size buckets, other arenas)."""
    from grotor_b200 import Router
    from grotor_b200.synth import WORKLOADS, Design
    small = Design(WORKLOADS["medium_320x320x10"].scaled(big_nets.nets.n, seed=46, two_pin_frac=1.0))
    assert small.nets.n == big_nets.nets.n
    ids = np.random.default_rng(1).permutation(small.nets.n).astype(np.int32)
    off = np.array([0, 7, 200, len(ids)], np.int32)

    def fresh(d):
        with Router(d.grid) as r:
            r.upload_nets(d.nets)
            r.set_plan(ids, off)
            return _stage(r, "plain")
    with Router(big_nets.grid) as r:
        r.upload_nets(small.nets)
        r.set_plan(ids, off)
        _stage(r, mode)
        r.upload_nets(big_nets.nets)
        _same(_stage(r, mode), fresh(big_nets))


def test_plan_of_nets_that_are_gone(big_nets):
    """Fewer nets than the plan names: every use of the plan is refused; a plan
    whose ids are all still there is not."""
    from grotor_b200 import GrbError, Router
    from grotor_b200.synth import WORKLOADS, Design
    d = big_nets
    few = Design(WORKLOADS["medium_320x320x10"].scaled(50, seed=47, two_pin_frac=1.0))
    with Router(d.grid) as r:
        r.upload_nets(d.nets)
        r.generate_batches_rsmt(d.order, 1000000)
        r.upload_nets(few.nets)
        for call in (lambda: r.lshape_route("plain"), lambda: r.lshape_route("graph"),
                     lambda: r.lshape_route("persistent"), lambda: r.route_batch(0, 1),
                     lambda: r.commit_batch_demand(0, 1, 1), lambda: r.autotune()):
            with pytest.raises(GrbError, match="no longer uploaded"):
                call()
        r.upload_nets(d.nets)
        r.set_plan(np.arange(40, dtype=np.int32), np.array([0, 40], np.int32))
        r.upload_nets(few.nets)
        assert r.lshape_route("plain")["wirelength"] > 0


@pytest.mark.parametrize("mode", ["plain", "graph", "persistent"])
def test_refused_planning_leaves_no_plan_behind(big_nets, mode):
    """A longer order than the plan's buffers hold, with an id that is not
    uploaded: the buffers grow, the call is refused, and a stage then has
    nothing to route."""
    from grotor_b200 import GrbError, Router
    d = big_nets
    with Router(d.grid) as r:
        r.upload_nets(d.nets)
        r.generate_batches_rsmt(d.order[:20], 1000000)
        bad = d.order.copy()
        bad[-1] = d.nets.n
        with pytest.raises(GrbError, match="out of range"):
            r.generate_batches_rsmt(bad, 1000000)
        ids, off = r.plan()
        assert len(ids) == 0 and off.tolist() == [0]
        assert r.lshape_route(mode)["wirelength"] == 0
        r.generate_batches_rsmt(d.order, 1000000)
        assert r.lshape_route(mode)["wirelength"] > 0


def test_upload_beyond_the_memory_leaves_no_nets_behind(big_nets):
    """An upload whose route storage no GPU holds (2^44 words) is refused and
    leaves the context without nets; a valid upload makes it usable again."""
    from dataclasses import replace
    from grotor_b200 import GrbError, Router
    from grotor_b200._abi import GRB_ENOMEM
    d = big_nets
    too_much = d.nets.route_off.copy()
    too_much[-1] = 1 << 44
    with Router(d.grid) as r:
        r.upload_nets(d.nets)
        r.generate_batches_rsmt(d.order, 1000000)
        want = _stage(r, "plain")
        ids, off = r.plan()
        with pytest.raises(GrbError) as e:
            r.upload_nets(replace(d.nets, route_off=too_much))
        assert e.value.code == GRB_ENOMEM
        r.reset()
        for call in (lambda: r.lshape_route("plain"), lambda: r.lshape_route("persistent"), lambda: r.route_batch(0, 1),
                     lambda: r.generate_batches_rsmt(d.order, 1000000)):
            with pytest.raises(GrbError):
                call()
        r.upload_nets(d.nets)
        r.set_plan(ids, off)
        _same(_stage(r, "plain"), want)


def test_refused_upload_with_less_route_storage(big_nets):
    """An invalid upload of more nets than before with less route storage (the
    buffers are replaced, then the trees are refused): a reset clears the storage
    there is, not the last upload's."""
    from grotor_b200 import GrbError, Router
    from grotor_b200.router import NetArrays
    d = big_nets
    n = 2 * d.nets.n
    z, e = np.zeros(n + 1, np.int32), np.zeros(0, np.int32)
    bad = NetArrays(np.arange(n + 1, dtype=np.int32), np.full(n, -1, np.int32), np.full(n, -1, np.int32),
                    np.zeros(n + 1, np.int64), z, e, z, e, z, e)
    with Router(d.grid) as r:
        r.upload_nets(d.nets)
        with pytest.raises(GrbError, match="outside the grid"):
            r.upload_nets(bad)
        r.reset()
        r.upload_nets(d.nets)
        r.generate_batches_rsmt(d.order, 1000000)
        assert r.lshape_route("plain")["wirelength"] > 0


@pytest.mark.parametrize("off", [[0, 60, 20, 40], [0, -1, 40], [0, 41, 40]])
def test_plan_offsets_that_decrease_are_refused(big_nets, off):
    from grotor_b200 import GrbError, Router
    with Router(big_nets.grid) as r:
        r.upload_nets(big_nets.nets)
        with pytest.raises(GrbError, match="must not decrease"):
            r.set_plan(np.arange(40, dtype=np.int32), np.array(off, np.int32))
        r.set_plan(np.arange(40, dtype=np.int32), np.array([0, 20, 20, 40], np.int32))
        assert r.lshape_route("plain")["wirelength"] > 0


def _modes_in_turn(r, run):
    """The graph executor under one wire-cost rule, the other, the first again:
    each equals the plain executor under that rule, and the rules differ."""
    want = {}
    for rule in (False, True):
        r.set_wire_cost_mode(rule)
        want[rule] = run("plain")
    assert not np.array_equal(want[False][0], want[True][0])
    for rule in (False, True, False):
        r.set_wire_cost_mode(rule)
        _same(run("graph"), want[rule])


def test_graph_after_a_wire_cost_mode_switch():
    from grotor_b200 import Router
    from grotor_b200.synth import WORKLOADS, Design
    d = Design(WORKLOADS["small_64x64x5"].scaled(2500, seed=48, cap_lo=1, cap_hi=4))
    with Router(d.grid) as r:
        r.upload_nets(d.nets)
        r.generate_batches_rsmt(d.order, 1000000)
        _modes_in_turn(r, lambda mode: _stage(r, mode))


def test_zshape_graph_after_a_wire_cost_mode_switch():
    from grotor_b200 import Router
    from grotor_b200.router import NetArrays
    from grotor_b200.synth import WORKLOADS, Design
    d = Design(WORKLOADS["small_64x64x5"].scaled(1500, seed=49, cap_lo=1, cap_hi=4))
    n, z = d.nets, d.zshape_trees()
    room = np.concatenate([[0], np.cumsum(1 + 64 * np.diff(z["node_off"]).astype(np.int64))])
    nets = NetArrays(n.node_off, n.nodes, n.parents, room, n.point_off, n.points, n.hseg_off, n.hsegs, n.vseg_off, n.vsegs)

    def run(mode):
        r.reset()
        st = r.zshape_route(mode)
        return r.read_routes(), r.read_tables()["demand_half"], st["wirelength"], st["vias"]
    with Router(d.grid) as r:
        r.upload_nets(nets)
        r.upload_zshape(z)
        r.generate_batches_rsmt(d.order, 1000000)
        r.plan_bbox_batches(250)
        _modes_in_turn(r, run)


def test_flt_graph_after_a_wire_cost_mode_switch():
    from grotor_b200 import Router
    g = load_golden("ref_flt_48x48x10_1500")
    dags, _, route2_off = flt_by_net(g)

    def run(mode):
        r.reset()
        st = r.flt_route(mode, remove_phase_one=False)
        routes = r.read_routes2()
        for a, b in zip(route2_off[:-1], route2_off[1:]):  # words behind a route's own are an earlier run's
            if b > a:
                routes[a + routes[a]:b] = 0
        return routes, r.read_tables()["demand_half"], st["wirelength"], st["vias"]
    with Router(golden_grid(g)) as r:
        r.upload_nets(golden_nets(g))
        r.upload_flt(dags, route2_off)
        r.set_plan(g["flt_batch_ids"], g["flt_batch_off"])
        _modes_in_turn(r, run)
