"""A scene whose curves are not in path order is refused as fast as a valid one
of its size is taken, and the handle goes on to render."""
import time

import numpy as np
import pytest

import spr

pytestmark = pytest.mark.gpu


def lines(pid, P):
    n = len(pid)
    pts = np.zeros((2 * n, 2), np.float32)
    pts[0::2] = np.c_[np.arange(n) % 97, np.arange(n) % 89]
    pts[1::2] = pts[0::2] + (1.5, 2.5)
    return spr.Scene(pts, np.repeat(pid, 2), 2 * np.arange(n), np.full(n, spr.CURVE_LINEAR), pid, np.zeros(n), np.zeros(P),
                     np.full(P, 0xFF808080))


@pytest.mark.parametrize("n", [100, 1 << 20])
def test_unordered_paths_are_refused_in_linear_time(n):
    good, bad = lines(np.arange(n), n), lines(np.arange(n) % 2 * (n - 1), n)
    with spr.VGRasterizer(96, 96, samples=8) as r:
        r.add_vg(good)  # (buffers and kernels are there)
        t = []
        for _ in range(3):
            t0 = time.perf_counter()
            r.add_vg(good)
            t1 = time.perf_counter()
            with pytest.raises(spr.SprError) as e:
                r.add_vg(bad)
            t.append((t1 - t0, time.perf_counter() - t1))
            assert e.value.status == spr.ERR_INVALID_SCENE
        # the same copies, checks and kernels; a pass over all paths for every curve
        # (5e11 writes, of 2 TB) would take several hundred times as long
        assert min(b for _, b in t) < 5 * min(g for g, _ in t) + 0.05
        r.add_vg(good)
        r.rasterize()
        image = r.read_image().copy()
    with spr.VGRasterizer(96, 96, samples=8) as r:
        r.add_vg(good)
        r.rasterize()
        assert np.array_equal(r.read_image(), image)
