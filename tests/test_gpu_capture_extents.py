"""Captured frames of odd pixel counts at every bounce count: each captured
array, the hits among them (16-byte entries), bit for bit against the oracle."""
import numpy as np
import pytest

import vrg
from helpers import compare_frame, params, terrain_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [2, 3, 4, 5, 6, 7, 8])
def test_capture_odd_pixel_counts(gpu_ctx, orc, nb):
    mats, n, world = terrain_world(7, 1, 1, 0.02)
    gpu_ctx.set_materials(mats, n)
    scene, objs = vrg.build_world(gpu_ctx, world)
    OW = orc.build_world(mats, n, world)
    try:
        for W, H in ((1, 1), (33, 31), (35, 2)):
            gr, orr = vrg.Renderer(gpu_ctx, W, H, nb), orc.Renderer(W, H, nb)
            for f in range(2):
                cam = vrg.orbit_camera(1, 1, 5 * f, 16, W, H)
                p = params(nee=1, view=0, spatial=2, nb=nb, seeds=(f, 30 + f, 60 + f))
                img, _ = gr.render_params(scene, cam, p, want_image=True)
                orr.render(OW, cam, p)
                diffs = compare_frame(gr, orr, nb)
                assert all(v == 0 for v in diffs.values()), (W, H, f, diffs)
                assert np.array_equal(img.reshape(-1), orr.image()[0].reshape(-1))
            gr.close()
            orr.close()
    finally:
        OW.close()
        scene.close()
        for o in objs:
            o.release()
