"""Saving and loading a renderer's state go through the renderer's own arrays, in
several parts where they are small (two bounces: 64 bytes per pixel, 80 needed).
Renderers of other bounce counts, whose parts end elsewhere, read and write the
same blob, and frames go on from it bit for bit."""
import numpy as np
import pytest

import vrg
from helpers import params, terrain_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(1, 1), (33, 31), (641, 411), (1024, 600)])
def test_state_goes_through_the_renderers_arrays(vrglib, W, H):
    ctx = vrg.Context(0)
    mats, n, blocks = terrain_world(7, 1, 1, 0.05)
    ctx.set_materials(mats, n)
    scene, objs = vrg.build_world(ctx, blocks)
    two, five = vrg.Renderer(ctx, W, H, 2), vrg.Renderer(ctx, W, H, 5)

    def frame(r, f):
        p = params(nee=1, view=1, spatial=2, nb=2, seeds=(f, 30 + f, 60 + f), slots=3, flags=0)
        return r.render_params(scene, vrg.orbit_camera(1, 1, 3 * f, 16, W, H), p, want_radiance=True)[1]
    try:
        for f in range(3):
            frame(two, f)
        frame(five, 0)
        blob = two.save_state()
        five.load_state(blob)
        assert np.array_equal(five.save_state(), blob)
        two.load_state(five.save_state())
        for f in range(3, 7):
            a, b = frame(two, f), frame(five, f)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), f
    finally:
        two.close()
        five.close()
        scene.close()
        for o in objs:
            o.release()
        ctx.close()
