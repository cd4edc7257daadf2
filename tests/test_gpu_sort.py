"""The per-path sort at the borders of its size classes (a warp, blocks of
256, 512 and 1,024 threads, chunks through global memory), with one block
class (few paths) and with all of them, against the CPU oracle."""
import numpy as np
import pytest

import oracle
import spr

pytestmark = pytest.mark.gpu

W, H = 640, 600


def path_of(n, rng):
    """Lines that give exactly n entries: vertical ones of 1 + crossings, the
    rest inside one cell; their columns in no order."""
    out = []
    while n > 0:
        k = int(min(n, rng.integers(1, 260)))
        x, y0 = rng.integers(0, W // 2) * 2 + 0.5, rng.integers(0, 40) * 2 + 0.5
        y1 = y0 + (2 * (k - 1) if k > 1 else 0.75)
        p = [(x, y0), (x + 0.25, y1)]
        out.append(p if rng.random() < 0.5 else p[::-1])
        n -= k
    return out


def scene_of(sizes, seed):
    rng = np.random.default_rng(seed)
    paths = [path_of(n, rng) for n in sizes]
    lines = [(p, ln) for p, path in enumerate(paths) for ln in path]
    v = np.asarray([pt for _, ln in lines for pt in ln], np.float32)
    pid = np.asarray([p for p, _ in lines], np.uint32)
    n = len(lines)
    return spr.Scene(v, np.repeat(pid, 2), np.arange(n) * 2, np.full(n, spr.CURVE_LINEAR), pid, np.zeros(n),
                     np.arange(len(sizes)) % 2, np.full(len(sizes), 0xB0302060))


SIZES = [0, 1, 2, 31, 32, 33, 511, 512, 513, 2047, 2048, 2049, 4095, 4096, 4097, 16383, 16384, 16385, 40000]


@pytest.mark.parametrize("tiny", [0, 400])
def test_segment_sizes(tiny):
    sizes = SIZES + [1 + k % 7 for k in range(tiny)]  # (with 400 more paths than SMs: all classes)
    scene = scene_of(sizes, 5 + tiny)
    ref = oracle.run(scene, W, H, samples=8)
    assert ref.counts["curve_fragment"] == sum(sizes)
    with spr.VGRasterizer(W, H, samples=8) as r:
        r.add_vg(scene)
        for sort in (1, 0, -1):
            r.set_tuning(sort=sort)
            r.rasterize()
            for st in ("SORT_PERM", "SORT_KEY", "WN_SCAN", "DRAW_LIST"):
                assert np.array_equal(r.dump(st), ref[st]), (sort, st)


@pytest.mark.parametrize("n", [20000, 100000])
def test_one_long_path(n):
    scene = scene_of([n], n)
    ref = oracle.run(scene, W, H, samples=8)
    with spr.VGRasterizer(W, H, samples=8) as r:
        r.add_vg(scene)
        r.rasterize()
        assert np.array_equal(r.dump("SORT_PERM"), ref["SORT_PERM"])
