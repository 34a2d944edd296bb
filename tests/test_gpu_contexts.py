"""Several contexts in one process: what one of them uploads or launches does not
change what another may launch (a kernel's limit of dynamic shared memory is the
process's, not a context's)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _zshape_router(n, seed, **kw):
    from grotor_b200 import Router
    from grotor_b200.router import NetArrays
    from grotor_b200.synth import WORKLOADS, Design
    pins = kw.pop("pins", 12)
    d = Design(WORKLOADS["small_64x64x5"].scaled(n, seed=seed, **kw), max_subnet_pins=pins)
    m, z = d.nets, d.zshape_trees()
    room = np.concatenate([[0], np.cumsum(1 + 64 * np.diff(z["node_off"]).astype(np.int64))])
    r = Router(d.grid)
    r.upload_nets(NetArrays(m.node_off, m.nodes, m.parents, room, m.point_off, m.points, m.hseg_off, m.hsegs,
                            m.vseg_off, m.vsegs))
    r.upload_zshape(z)
    r.generate_batches_rsmt(d.order, 1000000)
    r.plan_bbox_batches(250)
    return r, int(np.diff(z["node_off"]).max())


def _zroutes(r, mode):
    r.reset()
    r.zshape_route(mode)
    return r.read_routes()


@pytest.mark.parametrize("mode", ["plain", "graph", "persistent"])
def test_zshape_of_larger_trees_after_another_context(mode):
    """The first context's nets want more shared memory than the second's."""
    a, big = _zshape_router(300, 71, X=80, Y=72, cap_layers=10, two_pin_frac=0.1, geo_p=0.03, max_pins=64, pins=64,
                            bbox_median=30.0)
    with a:
        want = _zroutes(a, "persistent")
        b, small = _zshape_router(200, 72, two_pin_frac=1.0)
        with b:
            assert big > 48 and small < 8
            _zroutes(b, "plain")
            np.testing.assert_array_equal(_zroutes(a, mode), want)


def test_softmin_of_two_contexts_on_two_threads():
    """Contexts with different arenas, each on a thread of its own."""
    import torch
    from grotor_b200 import Router
    from grotor_b200.softmin import routing_cost
    from grotor_b200.synth import WORKLOADS, Design
    small = WORKLOADS["small_64x64x5"]
    designs = [Design(small.scaled(60, seed=73, cap_layers=10, two_pin_frac=0.1, geo_p=0.06, max_pins=20, bbox_median=20.0),
                      max_subnet_pins=20), Design(small.scaled(60, seed=74, cap_layers=3))]

    def cost(r, d):
        cap = torch.tensor(np.asarray(d.grid.capacity, np.float64).reshape(-1), device="cuda")
        return routing_cost(r, cap, torch.ones_like(cap), 2.0, 0.3).item()
    routers = [Router(d.grid) for d in designs]
    want = []
    for r, d in zip(routers, designs):
        r.upload_nets(d.nets)
        want.append(cost(r, d))
    got = [[], []]

    def work(k):
        for _ in range(40):
            try:
                got[k].append(cost(routers[k], designs[k]))
            except Exception as e:  # reported by the comparison below
                got[k].append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert got[k] == [want[k]] * 40
        routers[k].close()
