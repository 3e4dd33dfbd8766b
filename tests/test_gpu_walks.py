"""The persistent walks' work distribution and the light-hit collection at the
sizes where they can go wrong, bit for bit (0 ulp) against the oracle and
against the same frame without capture:
- queues shorter than a warp, a few entries short of one per resident warp and
  exactly one per warp, ending inside a warp's static share of 32, and
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
    (81, 60, 0, 8, 0.05),
    (76, 64, 0, 16, 0.05),
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


@pytest.mark.parametrize("offset,back,zoom", [
    ((0, 0, 0), 40.0, 1.0),
    ((4064, 2048, -4096), 40.0, 1.0),
    ((-4096, -4096, 4064), 900.0, 0.04),
    ((0, 0, 0), 940.0, 0.04),
    ((32, 0, -4064), 6.0, 2.0),
], ids=["origin", "corner", "corner-far", "far", "close"])
def test_box_margin_bit_exact(gpu_ctx, orc, offset, back, zoom):
    """The walks widen the traversal boxes by a margin worked out per ray from
    the magnitudes of the coordinates (ray_margin): worlds at the origin and at
    the far corners of the translation range, seen from near and from the other
    end of the ray range, along the axes (rays on block planes) and across."""
    W, H, nb = 160, 120, 4
    mats, n, world = terrain_world(11, 2, 2, 0.02)
    gpu_ctx.set_materials(mats, n)
    floor = np.zeros(vrg.CHUNK_BLOCKS, np.uint8)
    scene, up, OW, objs = vrg.Scene(gpu_ctx), vrg.SceneUploader(gpu_ctx), orc.World(mats, n), []
    gr, orr = vrg.Renderer(gpu_ctx, W, H, nb), orc.Renderer(W, H, nb)
    try:
        for cx in range(2):
            for cz in range(2):
                t = (offset[0] + 32 * cx, offset[1], offset[2] + 32 * cz)
                nbh = vrg.chunk_neighbours(world, cx, cz, floor)
                objs.append(up.upload_chunk(world[cx, cz], nbh))
                scene.add_object(2 * cx + cz, objs[-1], t)
                OW.add_chunk(2 * cx + cz, world[cx, cz], nbh, t)
        OW.commit()
        centre = np.array(offset, np.float64) + (32.0, 14.0, 32.0)
        for k, d in enumerate([(1.0, 0.0, 0.0), (0.0, 0.0, -1.0), (0.0, -1.0, 0.0), (0.6, -0.35, 0.7)]):
            d = np.array(d) / np.linalg.norm(d)
            side = np.cross(d, (0.0, -1.0, 0.0)) if abs(d[1]) < 0.9 else np.array((1.0, 0.0, 0.0))
            side /= np.linalg.norm(side)
            upv = np.cross(side, d)
            cam = vrg.Camera()
            cam.eye[:] = [float(np.float32(x)) for x in centre - d * (back + 32.0)]
            cam.front[:] = [float(np.float32(x)) for x in d]
            cam.right[:] = [float(np.float32(x)) for x in side * 0.55 * zoom]
            cam.up[:] = [float(np.float32(x)) for x in upv * 0.55 * zoom]
            cam.width, cam.height = W, H
            p = params(nee=1, view=0, nb=nb, seeds=(k, 5 + k, 9 + k))
            gr.render_params(scene, cam, p)
            orr.render(OW, cam, p)
            diffs = compare_frame(gr, orr, nb)
            assert all(v == 0 for v in diffs.values()), (k, diffs)
            assert gr.last_stats.error_flags == 0
    finally:
        OW.close()
        gr.close()
        scene.close()
