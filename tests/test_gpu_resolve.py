"""The resolve at the edges of its shared blending rounds, byte for byte
against the CPU oracle: cells of one entry, cells whose entries straddle a
round of 32 or pass the shared-memory ones, equal colours that merge, opaque
and invisible fills, every sample count and mode, gradient paints."""
import numpy as np
import pytest

import oracle
import spr

pytestmark = pytest.mark.gpu


def check(scene, W, H, **kw):
    ref = oracle.run(scene, W, H, **kw)
    with spr.VGRasterizer(W, H, **kw) as r:
        for width in (0, 8, 64):
            r.set_tuning(bin_width=width)
            r.add_vg(scene)
            r.rasterize()
            assert np.array_equal(r.read_image().reshape(-1), ref["IMAGE"]), width


@pytest.mark.parametrize("samples", [8, 16, 32])
@pytest.mark.parametrize("n_paths", [1, 2, 9, 40, 160])
@pytest.mark.parametrize("W,H", [(7, 5), (33, 18)])
def test_entries_per_cell(W, H, n_paths, samples):
    # every path over the whole small viewport: up to hundreds of partly
    # covering items per cell
    scene = spr.Scene.generate(spr.SCENE_RANDOM, seed=n_paths + W, width=W, height=H, n_paths=n_paths, seg_min=3,
                               seg_max=6)
    check(scene, W, H, samples=samples)


@pytest.mark.parametrize("alpha", [0, 1, 128, 254, 255])
@pytest.mark.parametrize("srgb", [True, False])
def test_alphas_and_equal_colours(alpha, srgb):
    # four colours in turn at one alpha: samples of different histories meet
    # in the same codes
    scene = spr.Scene.generate(spr.SCENE_RANDOM, seed=alpha, width=40, height=30, n_paths=60, seg_min=3, seg_max=5)
    scene.path_fill_rgba = (np.array([0x102030, 0x102030, 0xF0F0F0, 0x000000])[np.arange(60) % 4]
                            | (alpha << 24)).astype(np.uint32)
    check(scene, 40, 30, samples=32, srgb=srgb)


@pytest.mark.parametrize("samples,ms", [(8, True), (32, True), (16, False)])
def test_paints_between_solid_fills(samples, ms):
    scene = spr.Scene.generate(spr.SCENE_RANDOM, seed=9, width=36, height=26, n_paths=50, seg_min=3, seg_max=6)
    table = np.zeros((3, 12), np.uint32)
    f = table.view(np.float32)
    for i in range(3):
        f[i, 0:6] = (0.05, 0.01 * i, -0.8, -0.01, 0.06, -0.7)
        table[i, 6] = 256 * i
        f[i, 7] = 255 / 1024
        f[i, 8:11] = (0.1 * i, 0.2, 1 - 0.01 * i * i - 0.04)
    ramp = np.random.default_rng(3).integers(0, 1 << 32, 1024, dtype=np.uint64).astype(np.uint32)
    scene.path_fill_rgba[::2] = 1 + np.arange(25) % 3
    scene.gradients = (table.reshape(-1), ramp)
    check(scene, 36, 26, samples=samples, ms_output=ms)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 1024, 1025, 1500])
def test_items_per_bin(n):
    # n paths, each a triangle inside the one cell of the viewport: n items in
    # one bin, whose order decides the colours
    rng = np.random.default_rng(n)
    tri = rng.uniform(0.05, 1.95, (n, 3, 2))
    pts = tri[:, [0, 1, 1, 2, 2, 0]].reshape(-1, 2)
    pid = np.repeat(np.arange(n), 3)
    scene = spr.Scene(pts, np.repeat(pid, 2), 2 * np.arange(3 * n), np.full(3 * n, spr.CURVE_LINEAR), pid,
                      np.zeros(3 * n), np.zeros(n), rng.integers(0x10000000, 1 << 32, n).astype(np.uint32))
    check(scene, 2, 2, samples=32)
