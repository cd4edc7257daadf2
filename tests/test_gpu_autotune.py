"""The autotuner's resolve blocks per SM: below the default's, or the default."""
import pytest

import spr

pytestmark = pytest.mark.gpu


def test_resolve_blocks_are_not_the_default_under_another_name():
    # multisample resolves run 3 blocks per SM, so that 3 is no choice of its own;
    # a frame of a few microseconds, where noise decides between equal launches
    scene = spr.Scene.generate(spr.SCENE_LOCAL, seed=1, width=64, height=64, n_paths=4, seg_min=4, seg_max=8)
    with spr.VGRasterizer(64, 64, samples=8) as r:
        r.add_vg(scene)
        for _ in range(40):
            assert r.autotune(frames=1)["resolve_bps"] in (0, 2)
