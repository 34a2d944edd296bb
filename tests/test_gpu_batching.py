"""GPU first-fit batching equals the reference's CPU batching exactly.

The reference accepts RT-core batches only if the lists equal the CPU's
(generate_batches.hpp:113-131); the same bar applies to the grid kernels here,
in both execution forms, with small batch limits and sparsity > 1.
"""
import numpy as np
import pytest

import oracle
from helpers import golden_nets, load_golden

pytestmark = pytest.mark.gpu


def _check(router, order, nets, X, Y, limit, sparsity, mode):
    from grotor_b200 import plan_from_batches
    bo_ref, nb_ref = oracle.batches(X, Y, order, nets.point_off, nets.points, nets.hseg_off, nets.hsegs,
                                    nets.vseg_off, nets.vsegs, limit, sparsity)
    bo, nb = router.generate_batches_rsmt(order, limit, sparsity, mode)
    assert nb == nb_ref
    np.testing.assert_array_equal(bo, bo_ref)
    ids, off = router.plan()
    ids_ref, off_ref = plan_from_batches(order, bo_ref, nb_ref)
    np.testing.assert_array_equal(off, off_ref)
    np.testing.assert_array_equal(ids, ids_ref)


@pytest.mark.parametrize("mode", ["plain", "persistent"])
@pytest.mark.parametrize("limit,sparsity", [(1000000, 1), (37, 1), (1000000, 3), (1, 1)])
def test_synthetic(mode, limit, sparsity):
    from grotor_b200 import Router
    from grotor_b200.synth import WORKLOADS, Design
    d = Design(WORKLOADS["small_64x64x5"].scaled(3000 if limit > 1 else 700, seed=31))
    r = Router(d.grid)
    r.upload_nets(d.nets)
    _check(r, d.order, d.nets, d.grid.X, d.grid.Y, limit, sparsity, mode)
    r.close()


@pytest.mark.parametrize("mode", ["plain", "persistent"])
def test_medium_many_chunks(mode):
    """Several thousand nets across many 512-net chunks, big nets included."""
    from grotor_b200 import Router
    from grotor_b200.synth import WORKLOADS, Design
    d = Design(WORKLOADS["medium_320x320x10"].scaled(20000, seed=32))
    r = Router(d.grid)
    r.upload_nets(d.nets)
    _check(r, d.order, d.nets, d.grid.X, d.grid.Y, 1000000, 1, mode)
    r.close()


@pytest.mark.parametrize("mode", ["plain", "persistent"])
@pytest.mark.parametrize("n,limit", [(2500, 1000000), (2500, 3), (1250, 1000000), (240, 1000000)])
def test_nets_that_all_meet(n, limit, mode):
    """A grid so small that nearly every net meets every other: a colour per
    net or so (few and many words of colours), chains of conflicts as long as a
    chunk, with and without a tight limit."""
    from grotor_b200 import Router
    from grotor_b200.synth import WORKLOADS, Design
    d = Design(WORKLOADS["small_64x64x5"].scaled(n, seed=33, X=9, Y=8, bbox_median=4.0))
    r = Router(d.grid)
    r.upload_nets(d.nets)
    _check(r, d.order, d.nets, d.grid.X, d.grid.Y, limit, 1, mode)
    r.close()


@pytest.mark.parametrize("name", ["ref_64x64x10_2k", "ref_32x32x10_400"])
def test_reference_geometry(name):
    """On the reference's own FLUTE geometry the GPU reproduces the
    reference's batch lists."""
    from grotor_b200 import Router
    from helpers import golden_grid
    g = load_golden(name)
    grid, nets = golden_grid(g), golden_nets(g)
    r = Router(grid)
    r.upload_nets(nets)
    bo, nb = r.generate_batches_rsmt(g["order"], 1000000, 1, "persistent")
    np.testing.assert_array_equal(bo, g["batch_of"])
    ids, off = r.plan()
    np.testing.assert_array_equal(ids, g["ids"])
    np.testing.assert_array_equal(off, g["batch_off"])
    r.close()


def test_empty_and_single():
    from grotor_b200 import Router
    from grotor_b200.synth import WORKLOADS, Design
    d = Design(WORKLOADS["small_64x64x5"].scaled(50, seed=33))
    r = Router(d.grid)
    r.upload_nets(d.nets)
    bo, nb = r.generate_batches_rsmt(np.zeros(0, np.int32), 10)
    assert nb == 0 and len(bo) == 0
    bo, nb = r.generate_batches_rsmt(d.order[:1], 10)
    assert nb == 1 and bo.tolist() == [0]
    r.close()


@pytest.mark.parametrize("mode", ["plain", "persistent"])
def test_colours_that_run_out_only_on_the_way(mode):
    """256 colours, 254 of them taken by earlier nets that all meet.  Of the next
    chunk's nets a takes 254, e (meets a) 255, d (meets e) and b 254, c (meets b
    and d) 255.  While d still counts with 255, c has no colour left; the colouring
    that settles fits, so nothing is run again with more colours."""
    from grotor_b200 import Router
    from grotor_b200.router import GridArrays, NetArrays
    X, Y, L = 64, 64, 3
    g = GridArrays(L, X, Y, 1, 1.0, 2.0, np.ones(L), np.ones(X - 1, np.int32), np.ones(Y - 1, np.int32),
                   np.ones(L * X * Y, np.float32))
    row, meet = 40, 60  # the clique's marks run along y = row

    def nets(edges):
        points, marks = [], []
        for _ in range(254):
            points.append([2 * Y + 2])
            marks.append([(0 * Y + row, (X - 1) * Y + row)])
        while len(points) < 1024:  # the rest of the first chunk meets nothing
            points.append([(20 + 4 * (len(points) % 8)) * Y + 10 + 3 * (len(points) // 8 % 7)])
            marks.append([])
        names = "aedbc"
        for k, name in enumerate(names):
            points.append([4 * (k + 1) * Y + row])
            marks.append([])
        for k, (u, v) in enumerate(edges):  # v looks where u marks
            cell = 4 * (k + 1) * Y + meet
            marks[1024 + names.index(u)].append((cell, cell))
            points[1024 + names.index(v)].append(cell)
        n = len(points)
        off = lambda lists: np.cumsum([0] + [len(v) for v in lists]).astype(np.int32)
        z, e = np.zeros(n + 1, np.int32), np.zeros(0, np.int32)
        return NetArrays(z, e, e, np.zeros(n + 1, np.int64), off(points), np.concatenate(points).astype(np.int32), off(marks),
                         np.array([c for m in marks for s in m for c in s], np.int32), z, e)
    launches = []
    for edges in (["ae", "ed", "bc", "dc"], ["ae", "ed", "bc"]):
        m = nets(edges)
        order = np.arange(m.n, dtype=np.int32)
        with Router(g) as r:
            r.upload_nets(m)
            before = r.kernel_launches
            _check(r, order, m, X, Y, 1000000, 1, mode)
            launches.append(r.kernel_launches - before)
            colours, _ = oracle.batches(X, Y, order, m.point_off, m.points, m.hseg_off, m.hsegs, m.vseg_off, m.vsegs,
                                        1000000, 1)
            assert colours[-5:].tolist() == [254, 255, 254, 254, 255]
    assert launches[0] == launches[1]
