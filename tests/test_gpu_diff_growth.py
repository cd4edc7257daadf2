"""Growth of the adjoint's buffers: grown where a frame needs it, refused by a
memory limit without marking the handle."""
import numpy as np
import pytest

import oracle
import spr

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

REL_TOL = 1e-3  # (as the reference-gradient tests)


class Fit:
    """One scene's fill, gradient and outputs, and the oracle's."""

    def __init__(self, scene, W, H, samples, seed=3, alpha=(0.02, 0.6)):
        rng = np.random.default_rng(seed)
        self.scene = scene
        fill = np.c_[rng.uniform(0, 1, (scene.n_paths, 3)), rng.uniform(*alpha, (scene.n_paths, 1))].astype(np.float32)
        G = rng.normal(size=(H, W, 4)).astype(np.float32)
        self.ref_img, self.ref = oracle.diff(scene, W, H, fill, grad_image=G, samples=samples)
        self.fill, self.G = torch.tensor(fill, device="cuda"), torch.tensor(G, device="cuda")
        self.img = torch.zeros((H, W, 4), device="cuda")
        self.gf, self.gv = torch.zeros_like(self.fill), torch.zeros((scene.n_vertices, 2), device="cuda")

    def render(self, r):
        r.add_vg(self.scene)
        r.diff_render(self.fill.data_ptr(), self.img.data_ptr())

    def backward(self, r):
        r.diff_backward(self.fill.data_ptr(), self.G.data_ptr(), self.gf.data_ptr(), self.gv.data_ptr())

    def check(self):
        torch.cuda.synchronize()
        assert np.abs(self.img.cpu().numpy() - self.ref_img).max() < 1e-5
        for got, ref in ((self.gf, self.ref["fill"]), (self.gv, self.ref["vertex"])):
            assert np.linalg.norm(got.cpu().numpy() - ref) / max(np.linalg.norm(ref), 1e-30) < REL_TOL


def test_a_refused_growth_does_not_stick():
    """A cell of more than 64 fragments needs a deeper tape, which the limit
    refuses; a scene that fits the buffers held renders on the same handle."""
    W, H, S = 5, 4, 32
    small = Fit(spr.Scene.generate(spr.SCENE_RANDOM, seed=2, width=W, height=H, n_paths=3, seg_min=3, seg_max=4), W, H, S)
    deep = Fit(spr.Scene.generate(spr.SCENE_RANDOM, seed=3, width=W, height=H, n_paths=150, seg_min=3, seg_max=6), W, H, S)
    with spr.VGRasterizer(W, H, samples=S) as r:
        small.render(r)
        small.backward(r)  # the tape at its first depth: 8 blocks x 64 fragments x 16 KB
        deep.render(r)
        # room for the frame's other buffers, not for the doubled tape (16 MB in place of 10)
        r.set_memory_limit(r.frame_stats()["device_bytes"] + (3 << 20))
        with pytest.raises(spr.SprError) as e:
            deep.backward(r)
        assert e.value.status == spr.ERR_OUT_OF_MEMORY
        small.render(r)
        small.backward(r)
        small.check()
        r.set_memory_limit(0)
        for _ in range(2):  # (the growth, and with the grown tape)
            deep.render(r)
            deep.backward(r)
            deep.check()


def marks(n, x0, y0, w, rng):
    """n small quadrilaterals in the band of rows y0, y0 + 1: curves and paths."""
    pts, pid = [], []
    for p in range(n):
        cx, cy = x0 + rng.uniform(0.2, w - 0.2), y0 + rng.uniform(0.2, 1.8)
        q = [(cx - .15, cy - .15), (cx + .15, cy - .1), (cx + .1, cy + .15), (cx - .1, cy + .1)]
        for k in range(4):
            pts += [q[k], q[(k + 1) % 4]]
            pid.append(p)
    return pts, pid


def line_scene(pts, pid):
    m, n = len(pid), pid[-1] + 1
    return spr.Scene(np.asarray(pts, np.float32), np.repeat(pid, 2), 2 * np.arange(m), np.full(m, spr.CURVE_LINEAR), pid,
                     np.zeros(m), np.zeros(n), np.full(n, 0xFF808080))


def test_one_crowded_bin_under_a_limit():
    """4,096 paths in one bin of 8,192, some 130 to a cell: buffers by the items
    there are, not by the deepest bin for every warp.  (Under this limit the
    tape, 64 -> 256 fragments deep, is the largest: 800 MB.)"""
    W = H = 1024
    fit = Fit(line_scene(*marks(4096, 64, 100, 62, np.random.default_rng(0))), W, H, 8)
    with spr.VGRasterizer(W, H, samples=8) as r:
        r.set_memory_limit(1200 << 20)
        for _ in range(2):
            fit.render(r)
            fit.backward(r)
            fit.check()


@pytest.mark.parametrize("samples", [8, 32])
def test_crowded_band_among_empty_ones(samples):
    """500 slanted boxes along one band of a tall viewport, and 80 marks in one of
    its cells: bins of ten to twenty times the mean of items, and a tape that grows."""
    W, H = 192, 512
    rng = np.random.default_rng(4)
    pts, pid = [], []
    for p in range(500):
        x0, x1 = rng.uniform(-5, W * 0.3), rng.uniform(W * 0.6, W + 5)
        q = [(x0, 198), (x1, 198.5), (x1 - rng.uniform(0, 6), 204), (x0 + rng.uniform(0, 6), 204)]
        for k in range(4):
            pts += [q[k], q[(k + 1) % 4]]
            pid.append(p)
    pm, im = marks(80, 100, 200, 2, rng)
    fit = Fit(line_scene(pts + pm, pid + [500 + p for p in im]), W, H, samples)
    with spr.VGRasterizer(W, H, samples=samples) as r:
        fit.render(r)
        fit.backward(r)
        assert r.frame_stats()["host_syncs"] > 1  # (more than 64 fragments in a cell)
        fit.check()
        fit.render(r)
        fit.backward(r)
        assert r.frame_stats()["host_syncs"] == 1
        fit.check()


def covers(n, marked, W, H, rng):
    """n paths over the whole viewport and past it (a span in every cell row, no
    fragment), and after every `marked`-th of them a mark in some cell."""
    pts, pid, k = [], [], 0

    def add(q):
        nonlocal k
        for j in range(4):
            pts.extend([q[j], q[(j + 1) % 4]])
            pid.append(k)
        k += 1

    for p in range(n):
        add([(-7, -5), (W + 7, -5), (W + 7, H + 5), (-7, H + 5)])
        if marked and p % marked == marked - 1:
            x, y = rng.uniform(0.2, W - 0.2), rng.uniform(0.2, H - 0.2)
            add([(x - .15, y - .15), (x + .15, y - .1), (x + .1, y + .15), (x - .1, y + .1)])
    return line_scene(pts, pid)


@pytest.mark.parametrize("samples", [8, 16, 32])
@pytest.mark.parametrize("marked", [0, 1, 40, 300])
@pytest.mark.parametrize("n", [127, 128, 129, 256, 257, 513, 800])
def test_bins_in_parts(n, marked, samples):
    """Bins of up to 128 items and of two to thirteen times as many, which several
    warps go through in parts: cells without fragments, with fragments in every
    part, in some, in the last only.  (Alphas are small: the lowest layer counts.)"""
    W, H = 70, 3
    fit = Fit(covers(n, marked, W, H, np.random.default_rng(n)), W, H, samples, alpha=(0.001, 0.01))
    with spr.VGRasterizer(W, H, samples=samples) as r:
        for _ in range(2):
            fit.render(r)
            fit.backward(r)
            fit.check()
