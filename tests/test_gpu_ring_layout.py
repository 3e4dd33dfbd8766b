"""The reservoir ring's slots (pairs of planes, each slot at a 32-byte boundary):
the saved state keeps its order of five planes per slot, plane by plane the
captured reservoirs, and a renderer that loads it goes on bit for bit; odd
pixel counts, several parts of the copy, the staged spatial pass, and tuning
frames that leave the ring as it was."""
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


def _same(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("W,H,staging", [(1, 1, 0), (33, 31, 0), (33, 31, 1), (97, 64, 1), (641, 411, 0), (512, 512, 1)])
def test_saved_state_planes(gpu_ctx, world, W, H, staging):
    P, slots, nb = W * H, 3, 3
    a, b, c = (vrg.Renderer(gpu_ctx, W, H, nb) for _ in range(3))

    def frame(r, f, flags=0):
        p = params(nee=1, view=1, spatial=2, nb=nb, seeds=(f, 30 + f, 60 + f), slots=slots, flags=flags)
        return r.render_params(world, vrg.orbit_camera(2, 1, 3 * f, 16, W, H), p, want_radiance=True)[1]
    try:
        for r in (a, b):
            r.set_tuning(vrg.Tuning(spatial_staging=staging))
        temporal = []
        for f in range(slots):
            frame(a, f, vrg.RENDER_CAPTURE)
            temporal.append(a.readback(vrg.DBG_TEMPORAL, nb))
        blob = a.save_state()
        head = len(blob) - slots * 5 * P * 16 - P * 24
        ring = blob[head:head + slots * 5 * P * 16].view(np.float32).reshape(slots, 5, P, 4)
        for f, t in enumerate(temporal):  # (x_v n_v x_s n_s l p_omega seed ucw m w_sum)
            assert _same(ring[f, :, :, :3].transpose(1, 0, 2).reshape(P, 15), np.ascontiguousarray(t[:, :15])), f
            assert _same(np.ascontiguousarray(ring[f, :, :, 3].T), np.ascontiguousarray(t[:, [17, 19, 18, 15, 16]])), f
        b.load_state(blob)
        assert np.array_equal(b.save_state(), blob)
        c.load_state(blob)
        c.autotune(world, vrg.orbit_camera(2, 1, 0, 16, W, H),
                   params(nee=1, view=1, spatial=2, nb=nb, slots=slots, flags=0), frames=1)
        assert np.array_equal(c.save_state(), blob)
        for f in range(slots, slots + 4):
            ra = frame(a, f)
            assert _same(ra, frame(b, f)) and _same(ra, frame(c, f)), f
    finally:
        for r in (a, b, c):
            r.close()
