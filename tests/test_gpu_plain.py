"""Frames without reservoirs finish their pixels in the resolve pass: bit for
bit the plain view of the same frame with reservoirs (whose spatial pass
finishes them), over one and several bounces, odd extents, a scaled renderer,
capture, batched views and accumulation; the reservoir views read 0."""
import numpy as np
import pytest

import vrg
from helpers import params, terrain_world

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world(gpu_ctx):
    mats, n, blocks = terrain_world(7, 2, 1, 0.05)
    gpu_ctx.set_materials(mats, n)
    scene, objs = vrg.build_world(gpu_ctx, blocks)
    yield scene
    scene.close()


@pytest.mark.parametrize("W,H,nb,scale,flags", [
    (1, 1, 2, 1, 0),
    (257, 3, 3, 1, 0),
    (97, 61, 3, 1, vrg.RENDER_CAPTURE),
    (64, 48, 2, 2, 0),
    (33, 31, 8, 1, 0),
])
def test_plain_frames_equal_the_plain_view(gpu_ctx, world, W, H, nb, scale, flags):
    a, b = (vrg.Renderer(gpu_ctx, W, H, nb, scale=scale) for _ in range(2))
    try:
        for f in range(2):
            cam = vrg.orbit_camera(2, 1, 3 * f, 16, W, H)
            p = params(nee=1, view=0, spatial=2, nb=nb, seeds=(f, 30 + f, 60 + f), accumulate=int(scale == 1),
                       flags=flags)
            ia, ra = a.render_params(world, cam, p, want_image=True, want_radiance=True)
            p.flags = flags | vrg.RENDER_PLAIN_ONLY
            ib, rb = b.render_params(world, cam, p, want_image=True, want_radiance=True)
            assert np.array_equal(ia, ib) and np.array_equal(ra.view(np.uint32), rb.view(np.uint32))
        if scale == 1:
            (xa, na), (xb, n_b) = a.read_accumulation(), b.read_accumulation()
            assert na == n_b == 2 and np.array_equal(xa, xb)
        for view in (1, 2):
            p.debug_view = view
            ib, rb = b.render_params(world, cam, p, want_image=True, want_radiance=True)
            assert not rb.any()
    finally:
        a.close()
        b.close()


def test_one_bounce_and_batched(gpu_ctx, world):
    """One bounce has no reservoirs, with or without the flag, singly and in a batch."""
    ext = [(40, 30), (7, 5), (96, 17)]
    cams = [vrg.orbit_camera(2, 1, k, 16, w, h) for k, (w, h) in enumerate(ext)]
    for nb, flags in ((1, 0), (3, vrg.RENDER_PLAIN_ONLY), (3, vrg.RENDER_PLAIN_ONLY | vrg.RENDER_GRAPH)):
        br = vrg.BatchRenderer(gpu_ctx, ext, nb)
        try:
            p = params(nee=1, view=0, spatial=2, nb=nb, seeds=(1, 2, 3), flags=flags)
            imgs, rads = br.render([world] * 3, cams, p, [(5 + k, 9 + k) for k in range(3)], want_image=True,
                                   want_radiance=True)
            for k, (w, h) in enumerate(ext):
                r = vrg.Renderer(gpu_ctx, w, h, nb)
                q = params(nee=1, view=0, spatial=2, nb=nb, seeds=(1, 5 + k, 9 + k), flags=0)
                img, rad = r.render_params(world, cams[k], q, want_image=True, want_radiance=True)
                assert np.array_equal(imgs[k], img)
                assert np.array_equal(rads[k].view(np.uint32), rad.view(np.uint32))
                r.close()
        finally:
            br.close()
