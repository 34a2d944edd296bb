"""Measured cases of the routing path, each through the framework's public entry points.

A case is one pass of what a router's host program does with this library: a
whole routing stage (first-fit batching and the L-shape DAG), the same stage
one batch at a time, the default pipeline through its FLT stage, the GGR
pipeline's Z-shape stage, demand commits with the cost refresh they cause, the
topology build with the stage tail and the .out writer, and the differentiable
routing cost with its gradients.  Designs come from the repository's seeded
generator: the grids, net counts, pin and box distributions of its named
workloads, or sizes between them.

Every array a pass returns is what the program reads back: route words, batch
indices, cost tables, demand, flags, text, gradients.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from grotor_b200 import Router
from grotor_b200.router import GrbError, NetArrays
from grotor_b200.softmin import routing_cost
from grotor_b200.synth import WORKLOADS, Design, steiner_trees

LIMIT = 1000000      # nets per batch of the first-fit batching, as the stage drivers pass it
FLT_LIMIT = 300000   # the FLT stage's
BOX_LIMIT = 250      # the GGR pipeline's bounding-box batches
WORDS_PHASE2 = 1200  # phase-two route words per net (100 per pin, 12 pins)
ROOM = {"zshape": 330, "other": 44}  # route words per net a caller's buffer has room for
SHARE = {"commit": 0.6, "soft": 0.2}  # nets whose routes the caller brings
ABSENT = 1e30        # a candidate that does not exist (exact soft-min)


def listed():
    return [
        # A small block: the smallest stage a program routes, where latency and barriers count.
        {"name": "stage_small", "kind": "stage", "base": "small_64x64x5", "X": 64, "Y": 64, "layers": 5,
         "nets": 5000, "mode": "persistent"},
        # A ragged small grid (odd sides, an odd number of layers) through the per-batch launches.
        {"name": "stage_ragged", "kind": "stage", "base": "medium_320x320x10", "X": 149, "Y": 211, "layers": 7,
         "nets": 24000, "mode": "plain"},
        # An ordinary design: 120K nets on 320x320x10.
        {"name": "stage_medium", "kind": "stage", "base": "medium_320x320x10", "X": 320, "Y": 320, "layers": 10,
         "nets": 120000, "mode": "persistent"},
        # A large design: 900K nets on 800x800x10.
        {"name": "stage_large", "kind": "stage", "base": "large_800x800x10", "X": 800, "Y": 800, "layers": 10,
         "nets": 900000, "mode": "persistent"},
        # The largest grid, heavy-tailed pin counts and net lengths up to the whole die: the tables exceed L2.
        {"name": "stage_huge", "kind": "stage", "base": "persistent_1600x1600x10", "X": 1600, "Y": 1600, "layers": 10,
         "nets": 1500000, "mode": "persistent"},
        # The stage as a caller's own loop: refresh, route and commit per batch, then the tables.
        {"name": "seams_medium", "kind": "seams", "base": "medium_320x320x10", "X": 257, "Y": 301, "layers": 10,
         "nets": 60000},
        # Commits and a rip-up of routes the caller brings, and the cost tables after them.
        {"name": "commit_refresh", "kind": "commit", "base": "medium_320x320x10", "X": 397, "Y": 358, "layers": 10,
         "nets": 100000, "batches": 6},
        # The default pipeline through its detour stage: upload, L-shape, rip-up, FLT DAGs of the ripped-up nets.
        {"name": "flt_medium", "kind": "flt", "base": "medium_320x320x10", "X": 320, "Y": 320, "layers": 10,
         "nets": 120000, "mode": "persistent"},
        # The GGR pipeline: first-fit groups, bounding-box batches, Z-shape DP.
        {"name": "zshape_medium", "kind": "zshape", "base": "medium_320x320x10", "X": 320, "Y": 320, "layers": 10,
         "nets": 60000, "mode": "persistent"},
        # The differentiable cost, forward and gradients, in fp32 at a design's size ...
        {"name": "soft_f32", "kind": "soft", "base": "softmin_320x320x10", "X": 320, "Y": 320, "layers": 10,
         "nets": 120000, "dtype": "f32", "tau": 1.0},
        # ... and in fp64 on a ragged block.
        {"name": "soft_f64", "kind": "soft", "base": "softmin_320x320x10", "X": 73, "Y": 91, "layers": 8,
         "nets": 6000, "dtype": "f64", "tau": 0.1},
        # From Steiner trees to the written file: topology on the device, stage with its tail, .out text.
        {"name": "trees_to_out", "kind": "out", "base": "medium_320x320x10", "X": 200, "Y": 183, "layers": 10,
         "nets": 30000, "records": 2000},
    ]


def draw(rng):
    """One more case: sides 40 to 900, nets per 2-D cell as in the workloads."""
    kind = rng.choice(["stage", "stage", "stage", "seams", "commit", "flt", "zshape", "soft", "out"])
    top = {"stage": 900, "seams": 340, "commit": 500, "flt": 340, "zshape": 300, "soft": 340, "out": 260}[kind]
    X = int(round(math.exp(rng.uniform(math.log(40), math.log(top)))))
    Y = max(33, min(top, int(round(X * math.exp(rng.uniform(-0.6, 0.6))))))
    most = {"stage": 900000, "seams": 80000, "commit": 200000, "flt": 110000, "zshape": 55000, "soft": 110000,
            "out": 50000}[kind]
    nets = int(min(most, max(500, X * Y * rng.uniform(0.3, 1.3))))
    case = {"kind": kind, "X": X, "Y": Y, "nets": nets,
            "layers": 10 if kind == "flt" else rng.choice([5, 6, 7, 8, 9, 10, 10, 10, 10]),
            "base": rng.choice(["medium_320x320x10", "medium_320x320x10", "persistent_1600x1600x10"])}
    if kind in ("stage", "flt", "zshape"):
        case["mode"] = rng.choice(["persistent", "persistent", "plain"])
    if kind == "commit":
        case["batches"] = rng.randint(1, 9)
    if kind == "soft":
        case["base"] = "softmin_320x320x10"
        case["dtype"] = rng.choice(["f32", "f64"])
        case["tau"] = rng.choice([1.0, 0.1])
        if case["dtype"] == "f64":
            case["nets"] = min(nets, 30000)
    if kind == "out":
        case["records"] = rng.randint(200, 3000)
    return case


# ---- designs and inputs ----------------------------------------------------------------------------

class _Case:
    """The case's design: its base workload's distributions on the case's
    grid, cut to exactly case["nets"] routing subnets (splitting wide nets
    makes a few more than that)."""

    def __init__(self, case, seed):
        X, Y = case["X"], case["Y"]
        m = min(X, Y)
        d = Design(WORKLOADS[case["base"]].scaled(
            case["nets"], X=X, Y=Y, cap_layers=case["layers"], big_lo=max(2, m // 2), big_hi=max(3, m - 1),
            bbox_max=m, seed=int(seed) % (1 << 31) + 1))
        n, k = d.nets, case["nets"]
        self.grid = d.grid
        self.nets = NetArrays(
            n.node_off[:k + 1], n.nodes[:n.node_off[k]], n.parents[:n.node_off[k]], n.route_off[:k + 1],
            n.point_off[:k + 1], n.points[:n.point_off[k]], n.hseg_off[:k + 1], n.hsegs[:2 * n.hseg_off[k]],
            n.vseg_off[:k + 1], n.vsegs[:2 * n.vseg_off[k]])
        self.order = d.order[d.order < k]
        self.hpwl = d.hpwl[:k]
        if case["kind"] == "zshape":
            z = d.zshape_trees()
            e = z["node_off"][k]
            self.ztrees = {"node_off": z["node_off"][:k + 1], "coord": z["coord"][:e], "child": z["child"][:3 * e]}
        d.close()


def _design(case, seed):
    return _Case(case, seed)


def _pinned(case, words):
    """A caller-owned pinned buffer for the route words, with room to spare."""
    room = case["nets"] * (ROOM["zshape"] if case["kind"] == "zshape" else ROOM["other"]) + 4096
    return torch.zeros(max(int(words), room), dtype=torch.int32, pin_memory=True).numpy()


def _padded(a, size):
    """`a` with zeros behind it up to `size` entries."""
    out = np.zeros(max(size, len(a)), a.dtype)
    out[:len(a)] = a
    return out


def _ranks(group, n):
    """Position of every entry inside its group, in order (groups 0..n-1)."""
    order = np.argsort(group, kind="stable")
    start = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(group, minlength=n), out=start[1:])
    out = np.empty(len(group), np.int64)
    out[order] = np.arange(len(group)) - start[group[order]]
    return out


def _edges(grid, nets):
    """Every tree edge child -> parent: global child index, net, parent's global index, coordinates."""
    XY, Y = grid.X * grid.Y, grid.Y
    off = np.asarray(nets.node_off, np.int64)
    net_of = np.repeat(np.arange(nets.n), np.diff(off))
    par = np.asarray(nets.parents, np.int64)
    child = np.flatnonzero(par >= 0)
    p = off[net_of[child]] + par[child]
    nd = np.asarray(nets.nodes, np.int64)
    xy = nd % XY
    return child, net_of[child], p, xy[child] // Y, xy[child] % Y, xy[p] // Y, xy[p] % Y


def _own_routes(design, rng, share):
    """Routes a caller brings for a share of the nets (the others are not
    routed): every tree edge as an L on a horizontal and a vertical layer of
    the net, a via at the bend and one down to the pin."""
    g, n = design.grid, design.nets
    XY, Y, L = g.X * g.Y, g.Y, g.L
    child, net, p, x, y, px, py = _edges(g, n)
    routed = (rng.random(n.n) < share)[net]
    child, net, p, x, y, px, py = (v[routed] for v in (child, net, p, x, y, px, py))
    # A horizontal and a vertical layer per net, one above the other.
    lay = rng.integers(0, L - 1, n.n)
    first_h = ((lay & 1) ^ g.DIR) == 0
    h = np.where(first_h, lay, lay + 1)[net]
    v = np.where(first_h, lay + 1, lay)[net]
    pin = np.asarray(n.nodes, np.int64)[child] // XY
    entry = np.where(x != px, h, v)
    pairs = [
        (x != px, h * XY + np.minimum(x, px) * Y + y, h * XY + np.maximum(x, px) * Y + y),
        ((x != px) & (y != py), np.minimum(h, v) * XY + px * Y + y, np.maximum(h, v) * XY + px * Y + y),
        (y != py, v * XY + px * Y + np.minimum(y, py), v * XY + px * Y + np.maximum(y, py)),
        ((pin < L) & (pin != entry) & ((x != px) | (y != py)), np.minimum(pin, entry) * XY + x * Y + y,
         np.maximum(pin, entry) * XY + x * Y + y),
    ]
    owner = np.concatenate([net[m] for m, _, _ in pairs])
    a = np.concatenate([q[m] for m, q, _ in pairs])
    b = np.concatenate([q[m] for m, _, q in pairs])
    off = np.asarray(n.route_off, np.int64)
    at = off[owner] + 1 + 2 * _ranks(owner, n.n)
    routes = np.zeros(int(off[-1]), np.int32)
    routes[at] = a
    routes[at + 1] = b
    routes[off[:-1]] = 1 + 2 * np.bincount(owner, minlength=n.n)
    return routes, owner, a, b


def _flt_inputs(design, flags, count):
    """FLT DAGs of `count` nets: the flagged ones first, longest first, nets
    with a node of more than six children left out.  The tree's nodes; for every bent edge its
    two corners, competing for the parent's slot; and for bent edges of four
    cells and more each way the two runs that bend half way, two nodes each.
    With the batching geometry of those nets and their phase-two route
    offsets."""
    g, n = design.grid, design.nets
    XY, Y, L = g.X * g.Y, g.Y, g.L
    off = np.asarray(n.node_off, np.int64)
    size = np.diff(off)
    child, net, p, x, y, px, py = _edges(g, n)
    kids = np.bincount(p, minlength=int(off[-1]))
    most = np.maximum.reduceat(np.append(kids, 0), np.minimum(off[:-1], len(kids)))
    fit = (most <= 6) & (size >= 2)
    first = np.lexsort((np.arange(n.n), -design.hpwl.astype(np.int64), ~flags, ~fit))[:count]
    chosen = np.zeros(n.n, bool)
    chosen[first] = True
    chosen &= fit
    keep = chosen[net]
    child, net, p, x, y, px, py = (v[keep] for v in (child, net, p, x, y, px, py))
    slot = _ranks(p, int(off[-1]))
    bent = (x != px) & (y != py)
    long = bent & (abs(x - px) >= 4) & (abs(y - py) >= 4)
    local, plocal = child - off[net], p - off[net]
    # Depth: one more than the parent's for a straight edge, then one per node between.
    depth = np.zeros(int(off[-1]), np.int64)
    for i in range(1, int(local.max(initial=0)) + 1):
        m = local == i
        depth[child[m]] = depth[p[m]] + 1 + bent[m] + long[m]
    mx, my = (x + px) // 2, (y + py) // 2
    # Nodes between child and parent: (edges that have them, x, y, depth above the parent).
    between = [(bent, px, y, 1), (bent, x, py, 1), (long, mx, py, 1), (long, mx, y, 2), (long, px, my, 1),
               (long, x, my, 2)]
    e_at = np.concatenate([np.flatnonzero(m) for m, _, _, _ in between])
    b_net = net[e_at]
    b_local = size[b_net] + _ranks(b_net, n.n)
    b_cell = np.concatenate([L * XY + qx[m] * Y + qy[m] for m, qx, qy, _ in between])
    b_depth = depth[p[e_at]] + np.concatenate([np.full(int(m.sum()), k) for m, _, _, k in between])
    at = np.cumsum([0] + [int(m.sum()) for m, _, _, _ in between])
    corner_a, corner_b, low_h, high_h, low_v, high_v = (b_local[at[k]:at[k + 1]] for k in range(6))
    tree = np.flatnonzero(np.repeat(chosen, size))
    tree_net = np.repeat(np.arange(n.n), size)[tree]
    node_net = np.concatenate([tree_net, b_net])
    cell = np.concatenate([np.asarray(n.nodes, np.int64)[tree], b_cell])
    counts = np.bincount(node_net, minlength=n.n)
    node_off = np.concatenate([[0], np.cumsum(counts)])
    where = node_off[node_net] + np.concatenate([tree - off[tree_net], b_local])
    coord, dep, children = (np.zeros(int(node_off[-1]), np.int32) for _ in range(3))
    coord[where] = cell
    dep[where] = np.concatenate([depth[tree], b_depth])
    children[where] = np.concatenate([kids[tree], np.ones(len(b_net), np.int64)])
    # Edges (net, child, parent, slot at the parent), grouped by child node.
    st, zero = ~bent, np.zeros(len(child), np.int64)
    links = [(st, local[st], plocal[st], slot[st]),
             (bent, local[bent], corner_a, zero[bent]), (bent, local[bent], corner_b, zero[bent]),
             (bent, corner_a, plocal[bent], slot[bent]), (bent, corner_b, plocal[bent], slot[bent]),
             (long, local[long], high_h, zero[long]), (long, high_h, low_h, zero[long]),
             (long, low_h, plocal[long], slot[long]),
             (long, local[long], high_v, zero[long]), (long, high_v, low_v, zero[long]),
             (long, low_v, plocal[long], slot[long])]
    e_net = np.concatenate([net[m] for m, _, _, _ in links])
    e_child, e_par, e_slot = (np.concatenate([q[k] for q in links]) for k in (1, 2, 3))
    order = np.lexsort((np.arange(len(e_net)), e_child, e_net))
    e_net, e_child, e_par, e_slot = (v[order] for v in (e_net, e_child, e_par, e_slot))
    edge_off = np.concatenate([[0], np.cumsum(np.bincount(e_net, minlength=n.n))])
    per_node = np.bincount(node_off[e_net] + e_child, minlength=int(node_off[-1]))
    parent_end = np.cumsum(per_node) - np.repeat(edge_off[:-1], counts)
    dags = {"node_off": node_off, "coord": coord, "depth": dep, "children": children, "parent_end": parent_end,
            "edge_off": edge_off, "edge_parent": e_par, "edge_source_slot": e_child * 10 + e_slot}
    # Batching geometry: every DAG node's cell, every DAG edge's run.
    eu, ev = coord[node_off[e_net] + e_child] % XY, coord[node_off[e_net] + e_par] % XY
    lo, hi = np.minimum(eu, ev), np.maximum(eu, ev)
    hor, ver = eu // Y != ev // Y, (eu // Y == ev // Y) & (eu != ev)

    def segs(m):
        o = np.concatenate([[0], np.cumsum(np.bincount(e_net[m], minlength=n.n))]).astype(np.int32)
        return o, np.stack([lo[m], hi[m]], 1).astype(np.int32).reshape(-1)

    geometry = (node_off.astype(np.int32), (coord % XY).astype(np.int32), *segs(hor), *segs(ver))
    route2_off = np.concatenate([[0], np.cumsum(np.where(chosen, WORDS_PHASE2, 0))]).astype(np.int64)
    return chosen, dags, geometry, route2_off


def _stage_result(st):
    return np.array([st["wirelength"], float(st["vias"]), float(st["n_batches"]), float(st["stamp"])])


# ---- preparation -----------------------------------------------------------------------------------

def prepare(case, seed):
    d = _design(case, seed)
    g, n = d.grid, d.nets
    rng = np.random.default_rng(int(seed) & 0xffffffff)
    s = {"case": dict(case), "order": d.order}
    kind = case["kind"]
    if kind == "out":
        s["trees"] = steiner_trees(n, int(seed) % (1 << 31))
    if kind == "zshape":
        z = d.ztrees
        zn = np.diff(z["node_off"]).astype(np.int64)
        route_off = np.concatenate([[0], np.cumsum(1 + 64 * zn)]).astype(np.int64)
        n = NetArrays(n.node_off, n.nodes, n.parents, route_off, n.point_off, n.points, n.hseg_off, n.hsegs,
                      n.vseg_off, n.vsegs)
    r = Router(g)
    s["router"], s["nets"] = r, n
    r.upload_nets(n)
    s["routes"] = _pinned(case, n.route_off[-1])
    if kind == "zshape":
        r.upload_zshape(z)
        r.set_wire_cost_mode(True)
    elif kind == "seams":
        r.generate_batches_rsmt(d.order, LIMIT)
        s["ids"], s["off"] = r.plan()
    elif kind in ("commit", "soft"):
        s["own"] = _own_routes(d, rng, SHARE[kind])[0]
        nb = case.get("batches", 1)
        which = rng.integers(0, nb, n.n)
        s["ids"] = np.argsort(which, kind="stable").astype(np.int32)
        s["off"] = np.concatenate([[0], np.cumsum(np.bincount(which, minlength=nb))]).astype(np.int32)
        r.set_plan(s["ids"], s["off"])
        if kind == "soft":
            # The demand the gradients are taken at: the caller's routes, committed.
            r.write_routes_used(s["own"])
            for k in range(nb):
                r.commit_batch_demand(k, k + 1, 1)
            r.sync()
            dt = torch.float32 if case["dtype"] == "f32" else torch.float64
            cells = g.L * g.X * g.Y
            cap, uw, uv = _soft_inputs(g, rng, cells)
            s["cap"] = torch.tensor(cap, dtype=dt, device="cuda", requires_grad=True)
            s["uw"] = torch.tensor(uw, dtype=dt, device="cuda", requires_grad=True)
            s["uv"] = torch.tensor(uv, dtype=dt, device="cuda", requires_grad=True)
    elif kind == "flt":
        # The nets the pipeline's classification rips up, and if they are few the longest ones too.
        r.generate_batches_rsmt(d.order, LIMIT)
        r.lshape_route()
        chosen, s["dags"], s["geometry"], s["route2_off"] = _flt_inputs(d, r.ripup(0).astype(bool), max(20, n.n // 50))
        s["order2"] = d.order[chosen[d.order]]
    elif kind == "out":
        r.set_stage_tail(True, True, 0)
        k = min(case["records"], n.n)
        ids = rng.permutation(n.n)[:k].astype(np.int32)
        s["names"] = ["net%d" % i for i in ids]
        s["pins"] = [n.nodes[n.node_off[i]:n.node_off[i + 1]] for i in ids]
        s["extra"] = [np.zeros(0, np.int32)] * k
        s["subs"] = [ids[j:j + 1] for j in range(k)]
    r.sync()
    return s


def _soft_inputs(g, rng, cells):
    """Capacities near the design's, a unit wire cost per edge, a via cost."""
    cap = np.asarray(g.capacity, np.float64).reshape(-1)
    cap = np.where(cap > 0, cap + rng.uniform(-0.4, 0.4, cells), 0.0).astype(np.float32).astype(np.float64)
    uw = (g.unit_wire * rng.uniform(0.8, 1.2, cells)).astype(np.float32).astype(np.float64)
    return cap, uw, float(g.unit_via)


# ---- one pass ----------------------------------------------------------------------------------------

def run(s):
    return _RUN[s["case"]["kind"]](s)


def _run_stage(s):
    r, mode = s["router"], s["case"]["mode"]
    r.reset()
    batch_of, _ = r.generate_batches_rsmt(s["order"], LIMIT, 1, mode)
    st = r.lshape_route(mode)
    return {"batch_of": batch_of, "routes": r.read_routes(s["routes"]), "stats": _stage_result(st)}


def _run_seams(s):
    r = s["router"]
    r.reset()
    r.set_plan(s["ids"], s["off"])
    for b in range(len(s["off"]) - 1):
        r.refresh_cost()
        r.route_batch(b, b + 1)
        r.commit_batch_demand(b, b + 1, 1)
    r.refresh_cost()
    return {"routes": r.read_routes(s["routes"]), **r.read_tables()}


def _run_commit(s):
    r, nb = s["router"], len(s["off"]) - 1
    r.reset()
    r.write_routes_used(s["own"])
    for b in range(nb):
        r.refresh_cost()
        r.commit_batch_demand(b, b + 1, 1)
    r.refresh_cost()
    r.commit_batch_demand(nb - 1, nb + 1, -1)
    r.refresh_cost()
    return r.read_tables()


def _run_flt(s):
    r, mode = s["router"], s["case"]["mode"]
    r.reset()
    r.upload_nets(s["nets"])
    r.generate_batches_rsmt(s["order"], LIMIT, 1, mode)
    r.lshape_route(mode)
    flags = r.ripup(0)
    r.upload_geometry(*s["geometry"])
    r.upload_flt(s["dags"], s["route2_off"])
    batch_of, _ = r.generate_batches_rsmt(s["order2"], FLT_LIMIT, 1, mode)
    st = r.flt_route(mode, True)
    return {"flags": flags, "batch_of": batch_of, "routes": r.read_routes(s["routes"]), "routes2": r.read_routes2(),
            "stats": _stage_result(st)}


def _run_zshape(s):
    r, mode = s["router"], s["case"]["mode"]
    r.reset()
    batch_of, _ = r.generate_batches_rsmt(s["order"], LIMIT, 1, mode)
    r.plan_bbox_batches(BOX_LIMIT)
    try:
        st = r.zshape_route(mode)
    except GrbError:  # a net without a finite route: reported after the whole stage has run
        st = r.stats()
    return {"batch_of": batch_of, "routes": r.read_routes_used(s["routes"]), "stats": _stage_result(st)}


def _run_soft(s):
    cost = routing_cost(s["router"], s["cap"], s["uw"], s["uv"], s["case"]["tau"])
    dcap, duw, duv = torch.autograd.grad(cost, (s["cap"], s["uw"], s["uv"]))
    return {"cost": cost.detach(), "dcap": dcap, "duw": duw, "duv": duv}


def _run_out(s):
    r = s["router"]
    r.reset()
    r.build_topology(s["trees"])
    batch_of, _ = r.generate_batches_rsmt(s["order"], LIMIT)
    r.lshape_route()
    is_of, (cong, xsum, ysum) = r.stage_tail()
    text = r.write_out(s["names"], s["pins"], s["extra"], s["subs"])
    topo = r.read_topology()
    return {"batch_of": batch_of, "is_of": is_of, "congestion": cong, "xsum": xsum, "ysum": ysum,
            "text": _padded(np.frombuffer(text, np.uint8), 1000 * len(s["names"])),
            **{k: _padded(topo[k], 30 * len(s["order"]) + 4096) for k in ("nodes", "parents", "points", "hsegs", "vsegs")}}


_RUN = {"stage": _run_stage, "seams": _run_seams, "commit": _run_commit, "flt": _run_flt, "zshape": _run_zshape,
        "soft": _run_soft, "out": _run_out}


# ---- the work a pass cannot do without ---------------------------------------------------------------

def work(case):
    """Inputs read once and outputs written once: trees and batching geometry
    in, tables of the grid, route words out (about 3.4 tree nodes per net and
    8 route words per node, the generator's mean)."""
    n, cells = case["nets"], (case["layers"] - 1) * case["X"] * case["Y"]
    nodes = 3.4 * n
    topo = 8 * nodes + 4 * 2.5 * nodes + 8 * n
    routes = 4 * (1 * n + 8 * nodes)
    kind = case["kind"]
    if kind == "soft":
        b = 4 if case["dtype"] == "f32" else 8
        # Capacity, unit cost and demand in, two gradients out; about 9 * (9 + 45) candidates a tree edge, forward and
        # adjoint, of an exponential and two additions each.
        per_edge = (case["layers"] - 1) * 54 * 3 * 3
        return {"bytes": cells * (4 * b + 4) + 8 * nodes, "flops": per_edge * nodes}
    if kind == "commit":
        return {"bytes": routes + cells * (4 + 4 + 4 + 4 + 8 + 4), "flops": 0}
    tables = cells * 8  # capacity in, demand out
    if kind == "seams":
        tables += cells * 20
    return {"bytes": topo + routes + tables, "flops": 0}


# ---- tolerance and exact values ----------------------------------------------------------------------

def tolerance(case):
    """Whole numbers are equal.  The stages' routes follow from cost tables
    that the library defines bit for bit, so they are equal too.  Cost tables
    of a given demand hold float values of an fp32 exponential (seen: 1e-6);
    gradients are sums in the case's precision of soft minima whose arguments
    are divided by tau (seen: 7e-6 at tau 1 and 2.2e-5 at 0.1 in fp32, 9e-14
    in fp64; single values up to 3.6e-3 and 7e-12 of the mean)."""
    if case["kind"] == "commit":
        return {"rel": 4e-6, "max": 5e-6, "differ": 0.0}
    if case["kind"] == "soft":
        if case["dtype"] == "f32":
            return {"rel": 3e-5, "max": 4e-3} if case["tau"] >= 1 else {"rel": 1e-4, "max": 1.5e-2}
        return {"rel": 4e-13, "max": 3e-11}
    return "exact"


def exact(case, seed):
    if case["kind"] == "commit":
        return _exact_commit(case, seed)
    if case["kind"] == "soft":
        return _exact_soft(case, seed)
    return None


def _runs_to_cells(start, count, step):
    """Cells start, start + step, ... (count of them) of every run."""
    total = int(count.sum())
    first = np.repeat(np.cumsum(count) - count, count)
    k = np.arange(total) - first
    return np.repeat(start, count) + k * np.repeat(step, count)


def _commit(g, a, b, stamp, K, demand, ts):
    """Demand and timestamps after one batch's segments (a, b): wires first,
    then vias where no wire of the batch passes."""
    XY, Y = g.X * g.Y, g.Y
    la, lb = a // XY, b // XY
    w = la == lb
    wa, wb = a[w], b[w]
    ver = (wa % XY) // Y == (wb % XY) // Y
    step = np.where(ver, 1, Y)
    cells = _runs_to_cells(wa, (wb - wa) // step, step)
    demand += np.bincount(cells, minlength=len(demand)) * (2 * K)
    ts[cells] = stamp
    ts[wa] = stamp
    ts[wb] = stamp
    low, high = np.minimum(la, lb)[~w], np.maximum(la, lb)[~w]
    pos = (a % XY)[~w]
    c = _runs_to_cells(low * XY + pos, high - low, np.full(len(low), XY))
    c = c[ts[c] < stamp]
    l = c // XY
    ay = ((l & 1) ^ g.DIR) == 1
    along = np.where(ay, c % Y, c % XY // Y)
    length, stride = np.where(ay, Y, g.X), np.where(ay, 1, Y)
    head, tail = along == 0, along == length - 1
    mid = ~head & ~tail
    for cell, half in ((c[head], 2), ((c - stride)[tail], 2), ((c - stride)[mid], 1), (c[mid], 1)):
        demand += np.bincount(cell, minlength=len(demand)) * (half * K)


def _demand(d, case, rng, rip):
    """The caller's routes of the case committed (and its last batch ripped up)."""
    g, n = d.grid, d.nets
    _, owner, a, b = _own_routes(d, rng, SHARE[case["kind"]])
    nb = case.get("batches", 1)
    which = rng.integers(0, nb, n.n)
    demand = np.zeros(g.L * g.X * g.Y, np.int64)
    ts = np.zeros(len(demand), np.int64)
    for k in range(nb):
        m = which[owner] == k
        _commit(g, a[m], b[m], k + 1, 1, demand, ts)
    if rip:
        m = which[owner] == nb - 1
        _commit(g, a[m], b[m], nb + 1, -1, demand, ts)
    return demand, ts


def _exact_commit(case, seed):
    d = _design(case, seed)
    g = d.grid
    demand, ts = _demand(d, case, np.random.default_rng(int(seed) & 0xffffffff), True)
    dem = torch.as_tensor(demand, dtype=torch.float64).reshape(g.L, g.X, g.Y) * 0.5
    cap = torch.as_tensor(np.asarray(g.capacity, np.float64)).reshape(g.L, g.X, g.Y)
    uw = torch.full_like(cap, float(g.unit_wire))
    wc, vc, P = _soft_tables(g, dem, cap, uw, float(g.unit_via))
    return {"wcost": wc.numpy().reshape(-1), "vcost": vc.numpy().reshape(-1), "presum": P.numpy().reshape(-1),
            "demand_half": demand.astype(np.int32), "timestamp": ts.astype(np.int32)}


def _soft_tables(g, dem, cap, uw, uv):
    """Wire cost, via cost and exclusive wire-cost prefix along each track, in 64 bits."""
    L, X, Y = g.L, g.X, g.Y
    w = torch.as_tensor(np.asarray(g.short_costs, np.float64), device=cap.device).reshape(L, 1, 1)

    def over(dd):
        open_ = torch.exp(torch.minimum(0.5 * (dd - cap), g.of_cost_scale * 0.5 * (dd - cap)))
        shut = torch.exp(torch.minimum(1.5 * dd, g.of_cost_scale * 1.5 * dd))
        return torch.where(cap > 0.001, open_, torch.where(dd > 0, shut, torch.zeros_like(dd)))

    def incr(k):
        return torch.clamp((over(dem + k) - over(dem)) * w, max=1e12)

    one, half = incr(1.0), incr(0.5)
    xlen = torch.zeros(X, dtype=torch.float64, device=cap.device)
    ylen = torch.zeros(Y, dtype=torch.float64, device=cap.device)
    xlen[:X - 1] = torch.as_tensor(np.asarray(g.x_edge_len, np.float64))
    ylen[:Y - 1] = torch.as_tensor(np.asarray(g.y_edge_len, np.float64))
    wc, vc, P = [], [], []
    for l in range(L):
        dim = 1 if ((l & 1) ^ g.DIR) == 1 else 0
        m = Y if dim else X
        elen = ylen.reshape(1, Y) if dim else xlen.reshape(X, 1)
        wl = one[l] + uw[l] * elen
        v = torch.cat([one[l].narrow(dim, 0, 1), half[l].narrow(dim, 1, m - 2) + half[l].narrow(dim, 0, m - 2),
                       one[l].narrow(dim, m - 2, 1)], dim)
        c = torch.cumsum(wl, dim)
        P.append(torch.cat([torch.zeros_like(c.narrow(dim, 0, 1)), c.narrow(dim, 0, m - 1)], dim))
        wc.append(wl)
        vc.append(v + uv)
    return torch.stack(wc), torch.stack(vc), torch.stack(P)


def _exact_soft(case, seed):
    d = _design(case, seed)
    g, n = d.grid, d.nets
    rng = np.random.default_rng(int(seed) & 0xffffffff)
    demand, _ = _demand(d, case, rng, False)
    L, X, Y = g.L, g.X, g.Y
    XY = X * Y
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    cap, uw, uv = _soft_inputs(g, rng, L * XY)
    cap = torch.tensor(cap, device=dev, requires_grad=True)
    uw = torch.tensor(uw, device=dev, requires_grad=True)
    uv = torch.tensor(uv, dtype=torch.float64, device=dev, requires_grad=True)
    tau = case["tau"]
    dem = torch.as_tensor(demand, dtype=torch.float64, device=dev).reshape(L, X, Y) * 0.5
    _, vc, P = _soft_tables(g, dem, cap.reshape(L, X, Y), uw.reshape(L, X, Y), uv)
    vflat, pflat = vc.reshape(-1), P.reshape(-1)
    # Via stacks below each layer of a column: stack[l] = sum of vc[0..l-1].
    below = torch.cat([torch.zeros(1, X, Y, dtype=torch.float64, device=dev), torch.cumsum(vc, 0)]).reshape(L + 1, XY)

    def smin(v):
        return -tau * torch.logsumexp(-v / tau, -1)

    lo, hi = (torch.as_tensor(v, device=dev) for v in np.triu_indices(L))
    off = torch.as_tensor(np.asarray(n.node_off, np.int64), device=dev)
    nodes = torch.as_tensor(np.asarray(n.nodes, np.int64), device=dev)
    par = torch.as_tensor(np.asarray(n.parents, np.int64), device=dev)
    net = torch.repeat_interleave(torch.arange(n.n, device=dev), off[1:] - off[:-1])
    local = torch.arange(len(nodes), device=dev) - off[net]
    pin, xy = nodes // XY, nodes % XY
    x, y = xy // Y, xy % Y
    dist = (below[hi][:, xy] - below[lo][:, xy]).T
    gone = (pin < L)[:, None] & ((lo[None] > pin[:, None]) | (hi[None] < pin[:, None]))
    dist = torch.where(gone, torch.full_like(dist, ABSENT), dist)
    through = [torch.nonzero((lo <= l) & (hi >= l)).reshape(-1) for l in range(L)]
    ays = [((l & 1) ^ g.DIR) == 1 for l in range(L)]
    for i in range(int(local.max()), 0, -1):
        at = torch.nonzero(local == i).reshape(-1)
        p = off[net[at]] + par[at]
        cx, cy, px, py = x[at], y[at], x[p], y[p]
        x0, x1, y0, y1 = torch.minimum(cx, px), torch.maximum(cx, px), torch.minimum(cy, py), torch.maximum(cy, py)
        mine = dist[at]
        cur = torch.stack([smin(mine[:, t]) for t in through], 1)
        straight = (cx == px) | (cy == py)

        def wire(l, ax, ay_, bx, by):
            return pflat[l * XY + bx * Y + by] - pflat[l * XY + ax * Y + ay_]

        first, last, line = [], [], []
        for l in range(L):
            if ays[l]:
                first.append(wire(l, cx, y0, cx, y1))
                last.append(wire(l, px, y0, px, y1))
                line.append(torch.where(cx == px, first[l], torch.full_like(first[l], ABSENT)))
            else:
                first.append(wire(l, x0, cy, x1, cy))
                last.append(wire(l, x0, py, x1, py))
                line.append(torch.where(cy == py, first[l], torch.full_like(first[l], ABSENT)))
        ca, cb = cx * Y + py, px * Y + cy
        diag = []
        for pl in range(L):
            cand = []
            for cl in range(L):
                if cl == pl:
                    v = torch.where(straight, line[pl], torch.full_like(line[pl], ABSENT))
                elif (cl ^ pl) & 1:
                    corner = ca if ays[cl] else cb
                    a, b = min(cl, pl), max(cl, pl)
                    v = first[cl] + (below[b][corner] - below[a + 1][corner]) + last[pl]
                    v = torch.where(straight, torch.full_like(v, ABSENT), v)
                else:
                    continue
                cand.append(cur[:, cl] + v)
            diag.append(smin(torch.stack(cand, 1)))
        diag = torch.stack(diag, 1)
        add = torch.stack([smin(diag[:, a:b + 1]) for a, b in zip(lo.tolist(), hi.tolist())], 1)
        dist = dist.index_add(0, p, add)
    cost = smin(dist[off[:-1]]).sum()
    grads = torch.autograd.grad(cost, (cap, uw, uv))
    return {"cost": cost.detach().cpu(), "dcap": grads[0].cpu(), "duw": grads[1].cpu(), "duv": grads[2].cpu()}
