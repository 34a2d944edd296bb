"""The track-by-track cost refresh at the sizes where it can go wrong.

Routes brought by the caller (straight runs of every length on both kinds of
layer, via stacks, runs across their layer's direction) are committed in
batches and one batch is ripped up again; after every refresh the wire and via
costs equal a full recomputation of the demand with the device's exponential
bit for bit, the prefix table equals the oracle's prefix of them bit for bit,
and demand, timestamps and statistics equal the oracle's.  Grid sides cover one
bitmap word, a word's edge, a 128-position prefix block and its edges, a
1024-position window and its edges, and the longest track allowed.
"""
import numpy as np
import pytest

import oracle
from helpers import device_exp_table, orc_grid

pytestmark = pytest.mark.gpu

GRIDS = [(2, 2, 1, 0), (3, 33, 2, 1), (32, 31, 4, 1), (65, 64, 3, 0), (127, 128, 4, 1), (129, 40, 5, 1),
         (1023, 5, 2, 0), (1024, 1025, 2, 1), (7, 2100, 3, 1), (8192, 3, 2, 0)]


def _grid(X, Y, L, DIR, rng):
    from grotor_b200.router import GridArrays
    cap = rng.integers(0, 7, L * X * Y).astype(np.float32)
    return GridArrays(L, X, Y, DIR, 1.0, 2.0, 1.0 + rng.random(L), rng.integers(1, 9, X - 1).astype(np.int32),
                      rng.integers(1, 9, Y - 1).astype(np.int32), cap)


def _nets(g, n, rng, skew):
    """Route records of n nets (1-4 segments each)."""
    from grotor_b200.router import NetArrays
    XY = g.X * g.Y
    rec = []
    for _ in range(n):
        words = []
        for _ in range(int(rng.integers(1, 5))):
            l, x, y = int(rng.integers(g.L)), int(rng.integers(g.X)), int(rng.integers(g.Y))
            if rng.random() < 0.3 and g.L > 1:
                a, b = sorted(rng.integers(0, g.L, 2).tolist())
                words += [a * XY + x * g.Y + y, b * XY + x * g.Y + y]
                continue
            along_y = ((l & 1) ^ g.DIR) == 1
            if rng.random() < skew:
                along_y = not along_y
            size = g.Y if along_y else g.X
            span = min(size, int(2 ** rng.uniform(0, np.log2(size) + 0.5)))
            lo = int(rng.integers(0, size - span + 1))
            hi = lo + span - 1
            p, q = ((x, lo), (x, hi)) if along_y else ((lo, y), (hi, y))
            if rng.random() < 0.5:
                p, q = q, p
            words += [l * XY + p[0] * g.Y + p[1], l * XY + q[0] * g.Y + q[1]]
        rec.append([1 + len(words)] + words)
    off = np.cumsum([0] + [len(r) for r in rec]).astype(np.int64)
    z, e = np.zeros(n + 1, np.int32), np.zeros(0, np.int32)
    return NetArrays(z, e, e, off, z, e, z, e, z, e), np.concatenate(rec).astype(np.int32)


@pytest.mark.parametrize("skew", [0.0, 0.2])
@pytest.mark.parametrize("X,Y,L,DIR", GRIDS)
def test_refresh_equals_recomputation(X, Y, L, DIR, skew):
    from grotor_b200 import Router
    rng = np.random.default_rng(X * 31 + Y * 7 + L + DIR)
    g = _grid(X, Y, L, DIR, rng)
    n, nb = 90, 6
    nets, routes = _nets(g, n, rng, skew)
    order = rng.permutation(n).astype(np.int32)
    off = np.array([0, 1, 3, 10, 30, 60, n], np.int32)
    og = orc_grid(g)
    demand, ts = np.zeros(g.cells, np.int32), np.zeros(g.cells, np.int32)
    st = {"wirelength": 0.0, "vias": 0}
    with Router(g) as r, device_exp_table(og, 2 * 4 * n + 8):
        r.upload_nets(nets)
        r.set_plan(order, off)
        r.write_routes_used(routes)
        for step in range(nb + 2):
            r.refresh_cost()
            t = r.read_tables()
            w, v = oracle.cost_full(og, demand)
            for key, want in (("wcost", w), ("vcost", v), ("presum", oracle.presum(og, w)), ("demand_half", demand),
                              ("timestamp", ts)):
                np.testing.assert_array_equal(t[key], want, err_msg=f"{key} at step {step}")
            if step > nb:
                break
            b, k = (step, 1) if step < nb else (nb - 2, -1)
            r.commit_batch_demand(b, step + 1, k)
            oracle.commit_batch(og, order[off[b]:off[b + 1]], nets.route_off, routes, step + 1, k, demand, ts, st)
        s = r.stats()
        assert s["wirelength"] == st["wirelength"] and s["vias"] == st["vias"]


@pytest.mark.parametrize("X,Y", [(2500, 24), (8000, 16)])
def test_listed_refresh_of_the_persistent_stage(X, Y):
    """Grids with so many tracks that a persistent stage's CTAs list the dirty
    ones (below and above what is listed at once): routes, demand and costs
    equal the per-batch launches', which take every track in turn."""
    from grotor_b200 import Router
    from grotor_b200.synth import WORKLOADS, Design
    d = Design(WORKLOADS["small_64x64x5"].scaled(4000, seed=78, X=X, Y=Y, cap_layers=11, cap_lo=1, cap_hi=4))
    tracks = (d.grid.L + 1) // 2 * (X + Y)
    assert tracks > 5 * 2 * 148 * 8 and (tracks > 128 * 2 * 148) == (X > 7000)
    out = []
    with Router(d.grid) as r:
        r.upload_nets(d.nets)
        r.generate_batches_rsmt(d.order, 1000000)
        for mode in ("plain", "persistent"):
            r.reset()
            st = r.lshape_route(mode)
            r.refresh_cost()
            out.append((r.read_routes(), r.read_tables(), st["wirelength"], st["vias"]))
    (a, ta, wa, va), (b, tb, wb, vb) = out
    np.testing.assert_array_equal(a, b)
    for k in ta:
        np.testing.assert_array_equal(ta[k], tb[k])
    assert (wa, va) == (wb, vb)


@pytest.mark.parametrize("DIR", [0, 1])
def test_segments_between_two_tracks(DIR):
    """A caller's segment whose ends differ in x and in y, on layers of either
    direction: both end cells are stamped where they are, the edges are those
    along x at the first end's y, as the oracle commits them."""
    from grotor_b200 import Router
    from grotor_b200.router import NetArrays
    rng = np.random.default_rng(DIR)
    g = _grid(40, 37, 4, DIR, rng)
    XY, n = g.X * g.Y, 30
    rec = []
    for _ in range(n):
        l, (x0, x1), (y0, y1) = int(rng.integers(g.L)), rng.choice(g.X, 2, False), rng.choice(g.Y, 2, False)
        rec.append([3, l * XY + x0 * g.Y + y0, l * XY + x1 * g.Y + y1])
    routes = np.concatenate(rec).astype(np.int32)
    z, e = np.zeros(n + 1, np.int32), np.zeros(0, np.int32)
    nets = NetArrays(z, e, e, 3 * np.arange(n + 1, dtype=np.int64), z, e, z, e, z, e)
    og, ids = orc_grid(g), np.arange(n, dtype=np.int32)
    demand, ts = np.zeros(g.cells, np.int32), np.zeros(g.cells, np.int32)
    st = {"wirelength": 0.0, "vias": 0}
    with Router(g) as r:
        r.upload_nets(nets)
        r.set_plan(ids, np.arange(n + 1, dtype=np.int32))
        r.write_routes_used(routes)
        for b in range(n):
            r.commit_batch_demand(b, b + 1, 1)
            oracle.commit_batch(og, ids[b:b + 1], nets.route_off, routes, b + 1, 1, demand, ts, st)
        t = r.read_tables()
        np.testing.assert_array_equal(t["demand_half"], demand)
        np.testing.assert_array_equal(t["timestamp"], ts)
        assert r.stats()["wirelength"] == st["wirelength"]
