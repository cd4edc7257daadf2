"""Fill gradients of paths with very many fragments and spans: the sum over a
path's fragments and spans adds no error to their own."""
import numpy as np
import pytest

import oracle
import spr

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# A fragment's or span's share is the end of some ten roundings of 2^-24 (the
# blend, its adjoint, the sums over samples and over lanes).  Summed without
# further error, the gradients are off by no more than that.
REL_TOL = 10 * 2.0 ** -24


@pytest.mark.parametrize("samples", [8, 16, 32])
@pytest.mark.parametrize("paths,curves", [(1, 1500), (4, 400)])
def test_paths_of_many_fragments(paths, curves, samples):
    W = H = 512
    scene = spr.Scene.generate(spr.SCENE_RANDOM, seed=paths, width=W, height=H, n_paths=paths, seg_min=curves,
                               seg_max=curves)
    rng = np.random.default_rng(9)
    fill = np.c_[rng.uniform(0, 1, (paths, 3)), rng.uniform(0.3, 0.9, (paths, 1))].astype(np.float32)
    G = rng.normal(0.2, 1, size=(H, W, 4)).astype(np.float32)
    _, ref = oracle.diff(scene, W, H, fill, grad_image=G, samples=samples)
    with spr.VGRasterizer(W, H, samples=samples) as r:
        r.add_vg(scene)
        f, g = torch.tensor(fill, device="cuda"), torch.tensor(G, device="cuda")
        img = torch.empty((H, W, 4), device="cuda")
        gf, gv = torch.empty_like(f), torch.empty((scene.n_vertices, 2), device="cuda")
        r.diff_render(f.data_ptr(), img.data_ptr())
        r.diff_backward(f.data_ptr(), g.data_ptr(), gf.data_ptr(), gv.data_ptr())
        torch.cuda.synchronize()
    err = np.linalg.norm(gf.cpu().numpy() - ref["fill"]) / np.linalg.norm(ref["fill"])
    assert err <= REL_TOL, err
