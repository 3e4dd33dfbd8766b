"""The stage times of a frame with stats: every stage that ran has one, the
others read 0, and the stages of the main stream add up to no more than the
frame."""
import pytest

import vrg
from helpers import params, terrain_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,nb,flags", [
    (1, 1, 1, 0),
    (1, 1, 8, 0),
    (200, 113, 3, 0),
    (200, 113, 3, vrg.RENDER_CAPTURE),
    (640, 360, 8, 0),
])
def test_stage_times(gpu_ctx, W, H, nb, flags):
    mats, n, world = terrain_world(7, 2, 1, 0.02)
    gpu_ctx.set_materials(mats, n)
    scene, objs = vrg.build_world(gpu_ctx, world)
    r = vrg.Renderer(gpu_ctx, W, H, nb)
    try:
        for f in range(3):
            p = params(nee=1, view=1, spatial=1, nb=nb, seeds=(f, 30 + f, 60 + f))
            p.flags = flags
            r.render_params(scene, vrg.orbit_camera(2, 1, 3 * f, 16, W, H), p)
            st = r.last_stats
            for b in range(8):
                # (a bounce whose queue is empty shades nothing)
                ran = b < nb
                assert (st.ms_trace[b] > 0) == ran and st.ms_shade[b] >= 0, b
                assert st.ms_shade[b] == 0 if not ran else st.ms_shade[b] > 0 or W * H == 1, b
                assert (st.ms_anyhit[b] > 0) == (b + 1 < nb), b
                assert abs(st.ms_bounce[b] - st.ms_trace[b] - st.ms_shade[b]) < 1e-4
            assert st.ms_resolve > 0 and st.ms_spatial > 0
            # (the timer of the stages and the events' clock agree to a few us)
            assert sum(st.ms_bounce) + st.ms_resolve + st.ms_spatial <= st.ms_total + 0.005
    finally:
        r.close()
        scene.close()


def test_cache_frame_stage_times(gpu_ctx):
    """The training bounces of a cache frame run beside its main stream: their
    times start with the query bounce's light-pdf walk."""
    mats, n, world = terrain_world(7, 2, 1, 0.02)
    gpu_ctx.set_materials(mats, n)
    scene, objs = vrg.build_world(gpu_ctx, world)
    W, H = 320, 180
    r = vrg.Renderer(gpu_ctx, W, H, 8)
    cache = vrg.RadianceCache(gpu_ctx, (0.0, 0.0, 0.0), (64.0, 32.0, 32.0), seed=3)
    try:
        r.set_cache(cache)
        p = params(nee=1, view=1, spatial=1, nb=2, flags=vrg.RENDER_CACHE)
        p.cache_train_bounces = 4
        for f in range(3):
            r.render_params(scene, vrg.orbit_camera(2, 1, 3 * f, 16, W, H), p)
            st = r.last_stats
            assert st.error_flags == 0 and st.ms_resolve > 0 and st.ms_spatial > 0
            for b in range(8):
                assert (st.ms_trace[b] > 0) == (b < 6), b
                assert (st.ms_anyhit[b] > 0) == (b < 5), b
                assert 0 <= st.ms_shade[b] < st.ms_total and st.ms_trace[b] < st.ms_total
    finally:
        r.set_cache(None)
        cache.close()
        r.close()
        scene.close()
