"""The emission of intersection entries at the edges of its block layout,
against the CPU oracle: block sizes around the dispatch rule's steps, pieces
longer than one merge window, blocks whose crossings spill out of shared
memory, and coincident crossings (cell corners) across window borders."""
import numpy as np
import pytest

import oracle
import spr

pytestmark = pytest.mark.gpu


def scene_of(curves):
    """One path of the given curves ((type, points, weight) each)."""
    n = [len(p) for _, p, _ in curves]
    return spr.Scene(np.concatenate([np.asarray(p, np.float32) for _, p, _ in curves]), np.zeros(sum(n)),
                     np.cumsum([0] + n[:-1]), [t for t, _, _ in curves], np.zeros(len(curves)),
                     [w for _, _, w in curves], [0], [0xFF2040FF])


def check_entries(scene, W, H):
    ref = oracle.run(scene, W, H, samples=8)
    with spr.VGRasterizer(W, H, samples=8) as r:
        r.add_vg(scene)
        r.rasterize()
        for st in ("CURVE_COUNT", "INTERSECTION", "SORT_PERM", "DRAW_LIST"):
            assert np.array_equal(r.dump(st), ref[st]), st
    return ref.counts["curve_fragment"]


def curves_of(n, W, H, seed):
    rng = np.random.default_rng(seed)
    kinds = [spr.CURVE_LINEAR, spr.CURVE_QUADRATIC, spr.CURVE_CUBIC, spr.CURVE_RATIONAL]
    out = []
    for i in range(n):
        t = kinds[i % 4]
        out.append((t, rng.uniform((-20, -20), (W + 20, H + 20), (t & 7, 2)),
                    rng.uniform(0.2, 3)))
    return out


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 127, 128, 129, 6144, 6145, 12289])
def test_curve_counts_around_block_sizes(n):
    size = 300 if n < 1000 else 40
    check_entries(scene_of(curves_of(n, size, size, n)), size, size)


@pytest.mark.parametrize("kinds", range(1, 16))
def test_mixes_of_solvers(kinds):
    # every set of curve types: a block's lists of the three solvers empty,
    # partly filled and longer than a warp
    for n in (8, 64, 400):
        mix = [c for c in curves_of(4 * n, 120, 90, 100 * n + kinds)
               if kinds >> [spr.CURVE_LINEAR, spr.CURVE_QUADRATIC, spr.CURVE_CUBIC, spr.CURVE_RATIONAL].index(c[0]) & 1]
        check_entries(scene_of(mix[:n]), 120, 90)


@pytest.mark.parametrize("W,H", [(4096, 64), (64, 4096), (4095, 4093)])
def test_long_pieces_and_spilled_blocks(W, H):
    # (40 curves of thousands of crossings to a block: past its shared-memory buffer)
    nf = check_entries(scene_of(curves_of(40, W, H, W + H)), W, H)
    assert nf > 8 * 4096 or min(W, H) == 64


@pytest.mark.parametrize("length", [22, 24, 46, 48, 50, 130, 400])
def test_coincident_crossings_across_windows(length):
    # lines through cell corners: every crossing is of both directions, in
    # pieces just below and above the one-lane limit and a merge window
    c = []
    for x0, y0, sx, sy in [(0, 0, 1, 1), (length, 0, -1, 1), (0, 2, 1, 1), (2, length, 1, -1), (1, 1, 1, 1)]:
        c.append((spr.CURVE_LINEAR, [(x0, y0), (x0 + sx * length, y0 + sy * length)], 0.0))
        c.append((spr.CURVE_QUADRATIC, [(x0, y0), (x0 + sx * length / 2, y0 + sy * length / 2),
                                        (x0 + sx * length, y0 + sy * length)], 0.0))
        c.append((spr.CURVE_CUBIC, [(x0, y0), (x0 + sx * length / 4, y0 + sy * length / 4),
                                    (x0 + sx * 3 * length / 4, y0 + sy * 3 * length / 4),
                                    (x0 + sx * length, y0 + sy * length)], 0.0))
    # axis-parallel curves on and between cell lines: one chain only
    for k in (0, 1, 2, 2.5):
        c.append((spr.CURVE_LINEAR, [(k, 0), (k, length)], 0.0))
        c.append((spr.CURVE_CUBIC, [(0, k), (length / 3, k), (length / 2, k), (length, k)], 0.0))
    check_entries(scene_of(c), length + 3, length + 3)
