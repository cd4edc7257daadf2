"""A first frame that changes its resolve tile (short spans: 16 columns x 4 cell
rows in place of 64 x 1) in viewports where that makes more bins: the buffers
hold what the new tile needs."""
import numpy as np
import pytest

import oracle
import spr

pytestmark = pytest.mark.gpu


def marks(n, W, H, size, seed):
    """n quadrilaterals of `size` pixels: short spans or none."""
    rng = np.random.default_rng(seed)
    c = np.c_[rng.uniform(0, W, n), rng.uniform(0, H, n)]
    r = rng.uniform(0.3, 1, (n, 1, 1)) * size * np.array([[-1, -1], [1, -0.6], [0.6, 1], [-0.6, 0.6]]) / 2
    q = c[:, None, :] + r
    pts = np.stack([q, np.roll(q, -1, axis=1)], axis=2).reshape(-1, 2)
    pid = np.repeat(np.arange(n), 4)
    fill = (rng.integers(0, 1 << 24, n) | rng.integers(20, 200, n) << 24).astype(np.uint32)
    return spr.Scene(pts.astype(np.float32), np.repeat(pid, 2), 2 * np.arange(4 * n), np.full(4 * n, spr.CURVE_LINEAR), pid,
                     np.zeros(4 * n), np.zeros(n), fill)


# 2048 x 10: 160 bins of 64 columns, 256 of 16; 4096 x 2: 64 and 256; 640 x 42: 210 and 240
@pytest.mark.parametrize("W,H", [(2048, 10), (4096, 2), (640, 42)])
@pytest.mark.parametrize("samples", [8, 16, 32])
def test_many_entries_in_every_bin(W, H, samples):
    """More resolve warps than the first tile's bins, all of them with cells of
    more entries than stand in shared memory."""
    scene = marks(W * H // 2, W, H, 6.0, W)
    ref = oracle.run(scene, W, H, samples=samples)
    with spr.VGRasterizer(W, H, samples=samples) as r:
        r.add_vg(scene)
        for _ in range(2):
            r.rasterize()
            assert np.array_equal(r.read_image().reshape(-1), ref["IMAGE"])


def test_next_frames_allocate_nothing():
    """The frame after the change is captured, replayed, and runs under a memory
    limit of what the first one took."""
    W, H = 2048, 10
    scene = marks(20, W, H, 6.0, 1)
    ref = oracle.run(scene, W, H, samples=8, ms_output=False)
    for graph in (True, False):
        with spr.VGRasterizer(W, H, samples=8, ms_output=False) as r:
            r.set_graph_replay(graph)
            r.add_vg(scene)
            r.rasterize()
            held = r.frame_stats()["device_bytes"]
            r.set_memory_limit(held)
            for k in range(3):
                r.rasterize()
                assert r.frame_stats()["host_syncs"] == 0 and r.graph_replays() == (k + 1 if graph else 0)
                assert np.array_equal(r.read_image().reshape(-1), ref["IMAGE"])
            assert r.frame_stats()["device_bytes"] == held
