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

    def __init__(self, scene, W, H, samples, seed=3):
        rng = np.random.default_rng(seed)
        self.scene = scene
        fill = np.c_[rng.uniform(0, 1, (scene.n_paths, 3)), rng.uniform(0.02, 0.6, (scene.n_paths, 1))].astype(np.float32)
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
            assert np.linalg.norm(got.cpu().numpy() - ref) / np.linalg.norm(ref) < REL_TOL


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
