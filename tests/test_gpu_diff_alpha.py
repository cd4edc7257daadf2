"""Fill alphas outside [0, 1], which the composite takes as they are: a span's
1 - alpha is then negative or above 1, and so is the product over a run of
spans.  Image and gradients against the CPU reference gradient, in cells with
and without fragments, with one, two and many such spans in a run."""
import numpy as np
import pytest

import oracle
import spr

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# A layer rounds its sample states about three times (2^-24 each), and the
# layers above scale that by their |1 - alpha| <= 1.2: some 1e-5 of the largest
# state over the 40 layers here.  The gradients: as the reference-gradient tests.
IMG_TOL = 1e-4
REL_TOL = 1e-3

W, H = 130, 20
ALPHAS = {
    "one": [1.02],
    "one below zero": [-0.2],
    "pair": [1.5, 1.02],
    "under": [1.02, 0.3],
    "over": [0.3, 1.5],
    "three of five": [0.5, 1.5, 1.02, 0.7, 1.25],
    "mixed": [1.02, 0.4, -0.2, 0.6, 1.5, 0.3, 1.0, 0.8],
}


def boxes(n, rng):
    """n quadrilaterals across most of the viewport: cells with runs of spans,
    with and without fragments before, between and after them."""
    pts, pid = [], []
    for p in range(n):
        x0, x1 = rng.uniform(-5, W * 0.3), rng.uniform(W * 0.6, W + 5)
        y0, y1 = rng.uniform(-5, H * 0.4), rng.uniform(H * 0.6, H + 5)
        q = [(x0, y0), (x1, y0 + rng.uniform(0, 2)), (x1 - rng.uniform(0, 6), y1), (x0 + rng.uniform(0, 6), y1)]
        for k in range(4):
            pts += [q[k], q[(k + 1) % 4]]
            pid.append(p)
    m = len(pid)
    return spr.Scene(np.asarray(pts, np.float32), np.repeat(pid, 2), 2 * np.arange(m), np.full(m, spr.CURVE_LINEAR), pid,
                     np.zeros(m), np.zeros(n), np.full(n, 0xFF808080))


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("samples", [8, 16, 32])
@pytest.mark.parametrize("layers", [1, 3, 40])
@pytest.mark.parametrize("alphas", ALPHAS.values(), ids=ALPHAS.keys())
def test_alpha_outside_the_unit_range(alphas, layers, samples):
    n = max(layers, len(alphas))
    rng = np.random.default_rng(n)
    scene = boxes(n, rng)
    a = np.resize(alphas, n)
    if layers == 40:  # (a few of them among ordinary ones)
        a = np.where(np.arange(n) % 8 < len(alphas), a, 0.4)
    fill = np.c_[rng.uniform(0, 1, (n, 3)), a].astype(np.float32)
    G = rng.normal(size=(H, W, 4)).astype(np.float32)
    ref_img, ref = oracle.diff(scene, W, H, fill, grad_image=G, samples=samples)
    with spr.VGRasterizer(W, H, samples=samples) as r:
        r.add_vg(scene)
        f, g = torch.tensor(fill, device="cuda"), torch.tensor(G, device="cuda")
        img = torch.empty((H, W, 4), device="cuda")
        gf, gv = torch.empty_like(f), torch.empty((scene.n_vertices, 2), device="cuda")
        r.diff_render(f.data_ptr(), img.data_ptr())
        r.diff_backward(f.data_ptr(), g.data_ptr(), gf.data_ptr(), gv.data_ptr())
        torch.cuda.synchronize()
    assert np.abs(img.cpu().numpy() - ref_img).max() < IMG_TOL * max(1.0, np.abs(ref_img).max())
    assert rel(gf.cpu().numpy(), ref["fill"]) < REL_TOL
    assert rel(gv.cpu().numpy(), ref["vertex"]) < REL_TOL


def test_flat_cell_of_one_span():
    """Inside a box of fill (0.2, 0.4, 0.6, 1.02) on white: f a + c (1 - a)."""
    scene = spr.Scene(np.array([(10, 2), (100, 2), (100, 2), (100, 18), (100, 18), (10, 18), (10, 18), (10, 2)], np.float32),
                      np.zeros(8), 2 * np.arange(4), np.full(4, spr.CURVE_LINEAR), np.zeros(4), np.zeros(4), np.zeros(1),
                      np.full(1, 0xFF808080))
    fill = np.array([[0.2, 0.4, 0.6, 1.02]], np.float32)
    with spr.VGRasterizer(W, H, samples=8) as r:
        r.add_vg(scene)
        f = torch.tensor(fill, device="cuda")
        img = torch.empty((H, W, 4), device="cuda")
        r.diff_render(f.data_ptr(), img.data_ptr())
        torch.cuda.synchronize()
    assert np.abs(img.cpu().numpy()[10, 50] - (0.184, 0.388, 0.592, 1.0204)).max() < 1e-6
