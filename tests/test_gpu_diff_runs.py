"""The composite and its adjoint at the edges of their passes, against the CPU
reference gradient: cells without fragments and with many, runs of spans
across chunks of 32 items, bins of more items than the first span factors
hold, cells of more fragments than the first tape, odd widths."""
import numpy as np
import pytest

import oracle
import spr

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

REL_TOL = 1e-3  # (as the reference-gradient tests: both sides take the same crossings)


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


def check(scene, W, H, samples, seed):
    rng = np.random.default_rng(seed)
    P = scene.n_paths
    fill = np.c_[rng.uniform(0, 1, (P, 3)), rng.uniform(0.02, 0.6, (P, 1))].astype(np.float32)
    fill[::7, 3] = 1.0  # (opaque: nothing under them counts)
    G = rng.normal(size=(H, W, 4)).astype(np.float32)
    ref_img, ref = oracle.diff(scene, W, H, fill, grad_image=G, samples=samples)
    with spr.VGRasterizer(W, H, samples=samples) as r:
        r.add_vg(scene)
        f, g = torch.tensor(fill, device="cuda"), torch.tensor(G, device="cuda")
        img = torch.empty((H, W, 4), device="cuda")
        gf, gv = torch.empty_like(f), torch.empty((scene.n_vertices, 2), device="cuda")
        for _ in range(2):  # (again with the grown buffers)
            r.diff_render(f.data_ptr(), img.data_ptr())
            r.diff_backward(f.data_ptr(), g.data_ptr(), gf.data_ptr(), gv.data_ptr())
            torch.cuda.synchronize()
            assert np.abs(img.cpu().numpy() - ref_img).max() < 1e-5
            assert rel(gf.cpu().numpy(), ref["fill"]) < REL_TOL
            assert rel(gv.cpu().numpy(), ref["vertex"]) < REL_TOL


def boxes(n, W, H, rng):
    """n wide quadrilaterals with slanted sides: long runs of spans."""
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


@pytest.mark.parametrize("samples", [8, 16, 32])
@pytest.mark.parametrize("n,W,H", [(1, 65, 9), (3, 130, 20), (31, 66, 12), (33, 64, 12), (70, 127, 10), (300, 67, 11)])
def test_runs_of_spans(n, W, H, samples):
    check(boxes(n, W, H, np.random.default_rng(n)), W, H, samples, n)


@pytest.mark.parametrize("samples", [8, 16, 32])
def test_many_fragments_in_a_cell(samples):
    scene = spr.Scene.generate(spr.SCENE_RANDOM, seed=3, width=5, height=4, n_paths=150, seg_min=3, seg_max=6)
    check(scene, 5, 4, samples, 8)
