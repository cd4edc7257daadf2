"""The winding scan and marks at the edges of their tiles and warps, against the
CPU oracle: entry counts around a warp's and a tile's, with no items, fragments
only, and spans of one and of many bins."""
import numpy as np
import pytest

import oracle
import spr

pytestmark = pytest.mark.gpu


def lines(points):
    """Paths of closed polygons, one per entry of points."""
    v, pid, first, n = [], [], [], 0
    for k, poly in enumerate(points):
        for i in range(len(poly)):
            first.append(len(v))
            v += [poly[i], poly[(i + 1) % len(poly)]]
            pid.append(k)
    return spr.Scene(np.asarray(v, np.float32), np.repeat(pid, 2), first, [spr.CURVE_LINEAR] * len(pid), pid,
                     [0.0] * len(pid), [k % 2 for k in range(len(points))],
                     [0xFF2040FF + 977 * k & 0xFFFFFFFF | 0x80000000 for k in range(len(points))])


def check(scene, W, H, samples=8):
    ref = oracle.run(scene, W, H, samples=samples)
    with spr.VGRasterizer(W, H, samples=samples) as r:
        r.add_vg(scene)
        r.rasterize()
        for st in ("SORT_PERM", "DRAW_LIST", "MERGED_MASK"):
            assert np.array_equal(r.dump(st), ref[st]), st
        assert r.element_number() == ref.counts
    return ref.counts["curve_fragment"]


@pytest.mark.parametrize("where", ["inside", "outside"])
@pytest.mark.parametrize("n", [1, 84, 85, 1364, 1365, 2730])
def test_entries_around_warps_and_tiles(n, where):
    # triangles of three entries, one to a cell (outside: entries without items)
    W = H = 128
    dy = 0 if where == "inside" else H + 4
    tri = [[(2 * (k % 64) + a, 2 * (k // 64) + b + dy) for a, b in ((.2, .3), (1.7, .6), (.9, 1.8))] for k in range(n)]
    tri.append([(10.2, 10.3), (10.9, 10.4), (10.5, 10.9)])
    nf = check(lines(tri), W, H)
    assert where == "outside" or nf == 3 * (n + 1)


@pytest.mark.parametrize("W,H,rows", [(64, 520, 255), (300, 512, 256), (1100, 514, 257), (4096, 40, 16)])
def test_spans(W, H, rows):
    # a box of the viewport's width over `rows` cell rows and thin ones in it
    boxes = [[(1.3, 1.1), (W - 1.4, 1.1), (W - 1.4, 2 * rows - 1.2), (1.3, 2 * rows - 1.2)]]
    boxes += [[(x + .5, 3.5), (x + 5.5, 3.5), (x + 5.5, 2 * rows - 4.5), (x + .5, 2 * rows - 4.5)]
              for x in range(4, W - 8, max(W // 9, 8))]
    check(lines(boxes), W, H)


@pytest.mark.parametrize("samples", [8, 16, 32])
@pytest.mark.parametrize("n", [1, 2, 33, 127, 128, 200])
def test_groups_of_many_fragments(n, samples):
    # n nested triangles of one path in the last cell of the frame, and as many cells of one
    poly = []
    for k in range(n):
        e = .8 * k / n
        poly += [(62.1 + e, 62.2 + e), (63.9 - e / 9, 62.3 + e), (63 + e / 9, 63.9 - e / 9)]
    one = [[(2 * (k % 30) + .2, 2 * (k // 30) + .3), (2 * (k % 30) + 1.7, 2 * (k // 30) + .6),
            (2 * (k % 30) + .9, 2 * (k // 30) + 1.8)] for k in range(n)]
    check(lines(one + [poly]), 64, 64, samples)
