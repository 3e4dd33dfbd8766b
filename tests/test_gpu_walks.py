"""The persistent walks' work distribution and the light-hit collection at the
sizes where they can go wrong, bit for bit (0 ulp) against the oracle and
against the same frame without capture:
- queues shorter than a warp, ending inside a warp's static share of 32, and
  long enough that every warp takes further chunks (a grid of one CTA per SM);
- worlds with so many lamps that a ray sets aside more of them than its list
  holds, and crosses several (the sums of several hits)."""
import numpy as np
import pytest

import vrg
from helpers import compare_frame, params, terrain_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,grid,refill,emissive", [
    (1, 1, 0, 0, 0.01),
    (33, 1, 0, 32, 0.05),
    (96, 61, 0, 1, 0.3),
    (301, 173, 1, 8, 0.01),
    (301, 173, 1, 32, 0.3),
    (128, 96, 8, 3, 1.0),
])
def test_walks_bit_exact(gpu_ctx, orc, W, H, grid, refill, emissive):
    nb = 3
    mats, n, world = terrain_world(7, 2, 1, emissive)
    gpu_ctx.set_materials(mats, n)
    scene, objs = vrg.build_world(gpu_ctx, world)
    OW = orc.build_world(mats, n, world)
    gr, gp, orr = vrg.Renderer(gpu_ctx, W, H, nb), vrg.Renderer(gpu_ctx, W, H, nb), orc.Renderer(W, H, nb)
    try:
        for r in (gr, gp):
            r.set_tuning(vrg.Tuning(grid, refill, grid, grid, refill))
        for f in range(2):
            cam = vrg.orbit_camera(2, 1, 3 * f, 16, W, H)
            p = params(nee=1, view=1, spatial=3, nb=nb, seeds=(f, 30 + f, 60 + f))
            img, rad = gr.render_params(scene, cam, p, want_image=True, want_radiance=True)
            orr.render(OW, cam, p)
            oimg, orad = orr.image()
            diffs = compare_frame(gr, orr, nb)
            assert all(v == 0 for v in diffs.values()), (f, diffs)
            assert np.array_equal(img.reshape(-1), oimg.reshape(-1))
            p.flags = 0
            img2, _ = gp.render_params(scene, cam, p, want_image=True)
            assert np.array_equal(img, img2)
            assert gr.last_stats.error_flags == 0 and gp.last_stats.error_flags == 0
    finally:
        OW.close()
        gr.close()
        gp.close()
        scene.close()
