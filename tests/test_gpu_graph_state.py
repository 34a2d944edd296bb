"""A captured stage stays right when the context changes around it: scratch that
another executor has replaced by a larger one.  The plain executor, which
captures nothing, gives the expected routes."""
import numpy as np
import pytest

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
