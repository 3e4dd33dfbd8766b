"""Workloads of the framework for timing, each through the public interface of
vulkan-voxel-restir-gi_gb300/vrg.py and the C ABI it binds.

A case is a dict of plain values; its "kind" names the call:

  frame   one frame of one view of a terrain world (Renderer.render's work).
          out = "host": the blocking call that returns the packed image, as the
          reference's caller has it; out = "device": vrg_render without stats into
          device buffers, so that consecutive frames overlap, as a display or
          encoder loop on the GPU runs it.
  batch   one frame of many views of independent worlds (vrg_render_batched), in
          flight or replayed from the recorded launch sequence.
  cache   one frame whose paths end into the learned radiance cache.
  train   one training step of the radiance cache on the caller's samples.
  edit    an interactive edit: one chunk is uploaded anew, replaces the old one,
          and the next frame shows it.
  load    a world is uploaded, committed and shown for the first time.
"""
import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "vulkan-voxel-restir-gi_gb300"))
import vrg  # noqa: E402

AIR = 22      # the terrain's block types: 0-5 Lambertian, 6-21 emissive, 22 air
ORBIT = 64    # camera positions of one orbit around a world
BATCH_RES = [(256, 256), (640, 480), (1280, 720), (1920, 1080)]


def listed():
    return [
        # the smallest call: one chunk, a thumbnail, the image back on the host
        dict(name="thumb_64", kind="frame", nx=1, nz=1, width=64, height=64, bounces=2, nee=1, mode="parity",
             spatial=4, restir=True, mesh=False, emissive=0.01, out="host", radiance=False),
        # a small interactive window through the reference's own blocking call
        dict(name="window_640x480", kind="frame", nx=2, nz=2, width=640, height=480, bounces=3, nee=1,
             mode="parity", spatial=4, restir=True, mesh=False, emissive=0.005, out="host", radiance=False),
        # an odd extent with the player's rotated cube in view and the reference's
        # constants; the float image goes on to a denoiser on the device
        dict(name="mesh_957x541", kind="frame", nx=3, nz=5, width=957, height=541, bounces=4, nee=1, mode="parity",
             spatial=4, restir=True, mesh=True, emissive=0.01, out="device", radiance=True),
        # the benchmark's headline frame, frames in flight
        dict(name="restir_1080p", kind="frame", nx=4, nz=4, width=1920, height=1080, bounces=3, nee=1, mode="config",
             spatial=3, restir=True, mesh=False, emissive=0.005, out="device", radiance=False),
        # the ground-truth tracer: long paths without reuse, accumulated in FP64
        dict(name="truth_1080p", kind="frame", nx=8, nz=8, width=1920, height=1080, bounces=8, nee=1, mode="config",
             spatial=0, restir=False, mesh=False, emissive=0.005, out="device", radiance=True),
        # the largest single view: a large world at 4K with few, far lights
        dict(name="restir_4k", kind="frame", nx=16, nz=16, width=3840, height=2160, bounces=3, nee=1, mode="config",
             spatial=3, restir=True, mesh=False, emissive=0.002, out="device", radiance=True),
        # a server's batch: worlds and extents of all sizes in one launch sequence
        dict(name="batch_16", kind="batch", views=16, grid=8, top=3, bounces=2, emissive=0.005, graph=False),
        # many small views replayed from a recorded launch sequence, images to the host
        dict(name="batch_small_graph", kind="batch", views=24, grid=2, top=0, bounces=2, emissive=0.005, graph=True),
        # ReSTIR over paths that end into the learned cache
        dict(name="cache_1080p", kind="cache", nx=8, nz=8, width=1920, height=1080, levels=16, log2_table=19,
             train_bounces=4, emissive=0.005),
        # one training batch from the caller's own samples
        dict(name="train_65536", kind="train", n=65536, levels=16, log2_table=15),
        # a block is placed or dug in a world on screen
        dict(name="edit_720p", kind="edit", nx=8, nz=8, width=1280, height=720, bounces=3, emissive=0.005),
        # a world comes up: every chunk's mesh, lights and trees, and the first frame
        dict(name="load_8x8", kind="load", nx=8, nz=8, width=320, height=180, bounces=2, emissive=0.005),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "batch", "cache", "train", "edit", "load"])
    if kind == "frame":
        w = _log(rng, 64, 2600)
        restir = rng.random() < 0.8
        return dict(kind=kind, nx=rng.randint(1, 12), nz=rng.randint(1, 12), width=w,
                    height=max(40, int(w * rng.uniform(0.5, 0.8))),
                    bounces=rng.randint(2, 4) if restir else rng.randint(2, 8), nee=rng.choice([1, 1, 2, 0]),
                    mode=rng.choice(["parity", "config"]), spatial=rng.randint(1, 6) if restir else 0, restir=restir,
                    mesh=rng.random() < 0.25, emissive=rng.choice([0.002, 0.005, 0.01, 0.02]),
                    out=rng.choice(["host", "device", "device"]), radiance=rng.random() < 0.5)
    if kind == "batch":
        top = rng.randint(0, 3)
        return dict(kind=kind, views=rng.randint(2, [32, 24, 20, 12][top]), grid=rng.randint(1, 6), top=top,
                    bounces=rng.randint(2, 3), emissive=rng.choice([0.002, 0.005, 0.01]),
                    graph=rng.random() < 0.4)
    if kind == "cache":
        w = _log(rng, 480, 2200)
        return dict(kind=kind, nx=rng.randint(3, 10), nz=rng.randint(3, 10), width=w,
                    height=max(40, int(w * rng.uniform(0.5, 0.7))), levels=rng.choice([8, 12, 16]),
                    log2_table=rng.randint(15, 19), train_bounces=rng.randint(2, 5),
                    emissive=rng.choice([0.002, 0.005, 0.01]))
    if kind == "train":
        return dict(kind=kind, n=_log(rng, 1000, 65536), levels=rng.choice([8, 12, 16]),
                    log2_table=rng.randint(12, 15))
    if kind == "edit":
        w = _log(rng, 320, 1920)
        return dict(kind=kind, nx=rng.randint(3, 12), nz=rng.randint(3, 12), width=w, height=max(40, w * 9 // 16),
                    bounces=rng.randint(2, 3), emissive=rng.choice([0.002, 0.005, 0.01]))
    return dict(kind=kind, nx=rng.randint(1, 8), nz=rng.randint(1, 8), width=_log(rng, 64, 640),
                height=rng.randint(40, 360), bounces=2, emissive=rng.choice([0.002, 0.005, 0.01]))


_context = None


def _ctx():
    """The process's context with the terrain's materials, as a program makes it once."""
    global _context
    if _context is None:
        _context = vrg.Context(0)
        mats, n = vrg.terrain_materials(1)
        _context.set_materials(mats, n)
    return _context


def _rng(case, seed):
    return random.Random("%s %d" % (sorted(kv for kv in case.items() if kv[0] != "name"), seed))


def _cube(block):
    """A unit cube of 12 triangles around the origin, material slots 6 * block + face."""
    quads = [((0, 0, 0), (0, 0, 1), (0, 1, 1), (0, 1, 0)), ((1, 0, 0), (1, 1, 0), (1, 1, 1), (1, 0, 1)),
             ((0, 0, 0), (1, 0, 0), (1, 0, 1), (0, 0, 1)), ((0, 1, 0), (0, 1, 1), (1, 1, 1), (1, 1, 0)),
             ((0, 0, 0), (0, 1, 0), (1, 1, 0), (1, 0, 0)), ((0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))]
    uv = ((0.0, 0.0), (1.0, 0.0), (1.0, 1.0), (0.0, 1.0))
    v = np.zeros(36, vrg.VERTEX_DTYPE)
    k = 0
    for f, q in enumerate(quads):
        for i in (0, 1, 2, 0, 2, 3):
            v[k] = (np.array(q[i], np.float32) - np.float32(0.5), 6 * block + f, np.array(uv[i], np.float32))
            k += 1
    return v


def _world(ctx, nx, nz, emissive, seed):
    return vrg.build_world(ctx, vrg.terrain_blocks(seed, nx, nz, emissive))


def _params(case, st, flags=0):
    config = case.get("mode", "config") == "config"
    if not case.get("restir", True):
        flags |= vrg.RENDER_PLAIN_ONLY
    s = st["seed"] + 7919 * st["i"]
    return vrg.RenderParams(case.get("nee", 1), 1 if case.get("restir", True) else 0, case.get("spatial", 3),
                            case["bounces"], vrg.MODE_CONFIG if config else vrg.MODE_PARITY, s & 0x7fffffff,
                            (s + 1000) & 0x7fffffff, (s + 2000) & 0x7fffffff, 30.0 if config else 15.0,
                            20 if config else 0, 1 if config else 3,
                            1 if not case.get("restir", True) and config else 0, flags, case.get("train_bounces", 4))


def _camera(case, st):
    return vrg.orbit_camera(case["nx"], case["nz"], (st["at"] + st["i"]) % ORBIT, ORBIT, case["width"], case["height"])


def _device_outputs(st, w, h, radiance):
    st["bgra"] = torch.zeros(h, w, 4, dtype=torch.uint8, device="cuda")
    st["rad"] = torch.zeros(h, w, 3, dtype=torch.float32, device="cuda") if radiance else None
    torch.cuda.synchronize()  # the library's streams do not wait for torch's
    st["fo"] = vrg.FrameOutput(st["bgra"].data_ptr(), st["rad"].data_ptr() if radiance else None, vrg.OUTPUT_DEVICE, 0)


def _frame_state(case, seed):
    ctx, r = _ctx(), _rng(case, seed)
    scene, objs = _world(ctx, case["nx"], case["nz"], case["emissive"], r.randrange(1 << 30))
    if case.get("mesh"):
        a = r.uniform(0.2, 1.3)
        c, s = math.cos(a), math.sin(a)
        m = np.array([[c, 0, s, 16.0 * case["nx"]], [0, 1, 0, 27.0], [-s, 0, c, 16.0 * case["nz"]]], np.float32)
        cube = vrg.SceneUploader(ctx).upload_object(_cube(6 + r.randrange(16)))
        scene.add_object(1 << 20, cube, m)
        objs.append(cube)
    scene.commit()
    st = dict(case=case, scene=scene, objs=objs, i=0, at=r.randrange(ORBIT), seed=r.randrange(1 << 30))
    return ctx, r, st


def _samples(case, seed):
    """Surface points of an 8x8-chunk world with normals, directions and radiances."""
    g = np.random.default_rng(seed)
    n = case["n"]
    pos = (g.random((n, 3)) * np.array([256.0, 32.0, 256.0])).astype(np.float32)
    face = g.integers(0, 6, n)
    nrm = np.zeros((n, 3), np.float32)
    nrm[np.arange(n), face // 2] = np.where(face % 2, 1.0, -1.0)
    d = g.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    target = (np.abs(np.sin(pos[:, :1] * 0.2)) * np.array([[2.0, 1.0, 0.5]]) + 0.1).astype(np.float32)
    return pos, nrm, d, target


def _cache_values(case, seed):
    """Weights and table of a trained cache's magnitudes, exact in the working types (bf16, fp16)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn(vrg.NRC_MASTER, generator=g, device="cuda") * 0.17
    w[5 * 4096 + 3 * 64:] = 0
    t = torch.randn(case["levels"] << (case["log2_table"] + 1), generator=g, device="cuda") * 0.5
    return w.bfloat16().float().cpu().numpy(), t.half().float().cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        ctx, r, st = _frame_state(case, seed)
        st["renderer"] = vrg.Renderer(ctx, case["width"], case["height"], case["bounces"])
        if case["out"] == "device":
            _device_outputs(st, case["width"], case["height"], case["radiance"])
        return st
    if kind == "cache":
        ctx, r, st = _frame_state(case, seed)
        case = st["case"] = dict(case, bounces=2)
        # a trained cache that is held: the training work runs in every frame, its
        # step is too small to change the weights
        st["nrc"] = vrg.RadianceCache(ctx, (0, 0, 0), (32.0 * case["nx"], 32.0, 32.0 * case["nz"]),
                                      levels=case["levels"], log2_table=case["log2_table"], learning_rate=1e-30)
        w, t = _cache_values(case, r.randrange(1 << 30))
        st["nrc"].write(vrg.NRC_WEIGHTS, w)
        st["nrc"].write(vrg.NRC_TABLE, t)
        st["renderer"] = vrg.Renderer(ctx, case["width"], case["height"], 2 + case["train_bounces"])
        st["renderer"].set_cache(st["nrc"])
        _device_outputs(st, case["width"], case["height"], True)
        return st
    if kind == "batch":
        ctx, r = _ctx(), _rng(case, seed)
        n = case["views"]
        res = [BATCH_RES[v % (case["top"] + 1)] for v in range(n)]
        grids = [(r.randint(1, case["grid"]), r.randint(1, case["grid"])) for _ in range(n)]
        worlds = [_world(ctx, gx, gz, case["emissive"], r.randrange(1 << 30)) for gx, gz in grids]
        scenes = [s for s, _ in worlds]
        vrg.commit_scenes(scenes)
        st = dict(case=case, scenes=scenes, objs=[o for _, o in worlds], grids=grids, res=res, i=0,
                  at=r.randrange(ORBIT), seed=r.randrange(1 << 30), renderer=vrg.BatchRenderer(ctx, res, case["bounces"]))
        if not case["graph"]:
            st["rad"] = [torch.zeros(h, w, 3, dtype=torch.float32, device="cuda") for w, h in res]
            torch.cuda.synchronize()
            st["outs"] = (vrg.FrameOutput * n)()
            for v in range(n):
                st["outs"][v] = vrg.FrameOutput(None, st["rad"][v].data_ptr(), vrg.OUTPUT_DEVICE, 0)
        return st
    if kind == "train":
        r = _rng(case, seed)
        s = r.randrange(1 << 30)
        nrc = vrg.RadianceCache(_ctx(), (0, 0, 0), (256, 32, 256), levels=case["levels"],
                                log2_table=case["log2_table"], batch=case["n"])
        w, t = _cache_values(case, s)
        nrc.write(vrg.NRC_WEIGHTS, w)
        nrc.write(vrg.NRC_TABLE, t)
        return dict(case=case, nrc=nrc, samples=_samples(case, s))
    if kind == "edit":
        ctx, r, st = _frame_state(case, seed)
        nx, nz = case["nx"], case["nz"]
        # (the world's blocks as the game holds them; _frame_state drew its seed first)
        blocks = vrg.terrain_blocks(_rng(case, seed).randrange(1 << 30), nx, nz, case["emissive"])
        edits = []
        for _ in range(256):
            cx, cz, x, z = r.randrange(nx), r.randrange(nz), r.randrange(1, 31), r.randrange(1, 31)
            col = blocks[cx, cz].reshape(32, 32, 32)[x, :, z]
            top = int(np.argmax(col == AIR))
            edits.append((cx, cz, x, top if r.random() < 0.5 else top - 1, z, r.randrange(AIR), r.random() < 0.5))
        st.update(blocks=blocks, edits=edits, floor=np.zeros(vrg.CHUNK_BLOCKS, np.uint8),
                  up=vrg.SceneUploader(ctx), renderer=vrg.Renderer(ctx, case["width"], case["height"], case["bounces"]))
        return st
    if kind == "load":
        r = _rng(case, seed)
        return dict(case=case, i=0, at=r.randrange(ORBIT), seed=r.randrange(1 << 30),
                    world=vrg.terrain_blocks(r.randrange(1 << 30), case["nx"], case["nz"], case["emissive"]),
                    renderer=vrg.Renderer(_ctx(), case["width"], case["height"], case["bounces"]))
    raise ValueError(kind)


def _words(nodes):
    """A BvhNode array as its 32-bit words."""
    return nodes.view(np.int32).reshape(len(nodes), 10)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "train":
        nrc = state["nrc"]
        nrc.write(vrg.NRC_ZERO_GRADS)
        loss = nrc.train(*state["samples"], update=False)
        return dict(loss=loss, weight_grads=nrc.read(vrg.NRC_WEIGHT_GRADS), table_grads=nrc.read(vrg.NRC_TABLE_GRADS),
                    predictions=nrc.train_predictions())
    r = state["renderer"]
    if kind in ("frame", "cache"):
        p = _params(case, state, vrg.RENDER_CACHE if kind == "cache" else 0)
        cam = _camera(case, state)
        state["i"] += 1
        if case.get("out") == "host":
            img, rad = r.render_params(state["scene"], cam, p, want_image=True, want_radiance=case["radiance"])
            return dict(image=img, radiance=rad)
        vrg.check(r.ctx.lib.vrg_render(r.h, state["scene"].h, C.byref(cam), C.byref(p), C.byref(state["fo"]), None),
                  "vrg_render")
        return dict(image=state["bgra"], radiance=state["rad"])
    if kind == "batch":
        n, s = case["views"], state["seed"] + 7919 * state["i"]
        cams = [vrg.orbit_camera(gx, gz, (state["at"] + state["i"] + 5 * v) % ORBIT, ORBIT, w, h)
                for v, ((gx, gz), (w, h)) in enumerate(zip(state["grids"], state["res"]))]
        seeds = [((s + 2 * v) & 0x7fffffff, (s + 2 * v + 1) & 0x7fffffff) for v in range(n)]
        p = _params(case, state, vrg.RENDER_GRAPH if case["graph"] else vrg.RENDER_NO_PACK)
        # a recorded launch sequence serves frames of equal parameters: the views carry the seeds
        p.raygen_seed, p.temporal_seed, p.spatial_seed = 0, 0, 0
        state["i"] += 1
        if case["graph"]:
            imgs, _ = r.render(state["scenes"], cams, p, seeds, want_image=True)
            return imgs
        views = (vrg.View * n)()
        for v in range(n):
            views[v] = vrg.View(state["scenes"][v].h, cams[v], *seeds[v])
        vrg.check(r.ctx.lib.vrg_render_batched(r.h, views, n, C.byref(p), C.cast(state["outs"], C.c_void_p), None),
                  "vrg_render_batched")
        return state["rad"]
    if kind == "edit":
        cx, cz, x, y, z, block, dig = state["edits"][state["i"] % len(state["edits"])]
        blocks, nz, scene = state["blocks"], case["nz"], state["scene"]
        blocks[cx, cz].reshape(32, 32, 32)[x, y, z] = AIR if dig else block
        obj = state["up"].upload_chunk(blocks[cx, cz], vrg.chunk_neighbours(blocks, cx, cz, state["floor"]))
        key = cx * nz + cz
        scene.remove_object(key)
        scene.add_object(key, obj, (32 * cx, 0, 32 * cz))
        state["objs"][key] = obj
        cam, p = _camera(case, state), _params(case, state)
        state["i"] += 1
        return r.render_params(scene, cam, p)[0]
    scene, objs = vrg.build_world(r.ctx, state["world"])
    light, geo = scene.get_tlas()
    cam, p = _camera(case, state), _params(case, state)
    state["i"] += 1
    img, _ = r.render_params(scene, cam, p)
    info = np.array([list(o.info().values()) for o in objs], np.int64)
    scene.close()
    return dict(light_tree=_words(light), geometry_tree=_words(geo), info=info, image=img)


# bytes a surface block of a world cannot do without: its place, faces and block id
_BLOCK = 16


def _pixels(case):
    if case["kind"] == "batch":
        return sum(w * h for w, h in (BATCH_RES[v % (case["top"] + 1)] for v in range(case["views"])))
    return case["width"] * case["height"]


def work(case):
    if case["kind"] == "train":
        n, words = case["n"], case["levels"] << (case["log2_table"] + 1)
        # samples in, table and gradients; forward, and both halves of the backward
        return dict(bytes=48 * n + 12 * n + 6 * words + 8 * vrg.NRC_MASTER, flops=3 * 2 * n * (5 * 64 * 64 + 3 * 64))
    P, nb = _pixels(case), case.get("bounces", 2)
    if case["kind"] == "batch":
        blocks = 1200 * case["views"] * ((case["grid"] + 1) / 2) ** 2
    else:
        blocks = 1200 * case["nx"] * case["nz"]
    # per pixel: the reservoir read and written and the image; the world once
    restir = case.get("restir", True)
    per_pixel = (160 if restir else 0) + 4 + (12 if case.get("radiance") or case["kind"] in ("batch", "cache") else 0)
    if not restir and case.get("mode") == "config":
        per_pixel += 48  # the FP64 sum
    # a vertex: one face hit, its frame and material, one sampled direction and its pdf
    flops = 150 * P * nb
    size = per_pixel * P + _BLOCK * blocks
    if case["kind"] == "load":
        size += 32768 * case["nx"] * case["nz"]
    if case["kind"] == "cache":
        flops += 2 * P * (5 * 64 * 64 + 3 * 64) + 3 * 2 * 65536 * (5 * 64 * 64 + 3 * 64)
        size += 2 * (case["levels"] << (case["log2_table"] + 1))
    return dict(bytes=size, flops=flops)


def exact(case, seed):
    """A training step in 64 bits: a hash grid (trilinear over the cell's 8 corners),
    octahedral normal and view direction, a 5 x 64 ReLU network and the relative L2
    loss.  A frame has no such value: its random paths branch on every rounding."""
    if case["kind"] != "train":
        return None
    s = _rng(case, seed).randrange(1 << 30)
    w, t = _cache_values(case, s)
    pos, nrm, d, target = (torch.from_numpy(a).cuda().double() for a in _samples(case, s))
    L, T, n = case["levels"], 1 << case["log2_table"], case["n"]
    W = torch.from_numpy(w).cuda().double().requires_grad_(True)
    table = torch.from_numpy(t).cuda().double().reshape(L, T, 2).requires_grad_(True)
    p = (pos / torch.tensor([256.0, 32.0, 256.0], device="cuda", dtype=torch.float64)).clamp(0, 1)
    growth = math.exp((math.log(2048.0) - math.log(16.0)) / (L - 1))
    feats = []
    for level in range(L):
        res = math.floor(16 * math.pow(growth, level))
        g = p * res
        c = g.floor()
        f, c = g - c, c.long()
        out = 0
        for k in range(8):
            o = torch.tensor([(k >> 2) & 1, (k >> 1) & 1, k & 1], device="cuda")
            q = c + o
            if (res + 1) ** 3 <= T:
                ix = (q[:, 0] + q[:, 1] * (res + 1) + q[:, 2] * (res + 1) ** 2) & (T - 1)
            else:
                ix = (q[:, 0] ^ (q[:, 1] * 2654435761) ^ (q[:, 2] * 805459861)) & (T - 1)
            wk = torch.where(o == 1, f, 1 - f).prod(1)
            out = out + wk[:, None] * table[level][ix]
        feats.append(out)

    def octahedral(v):
        xy = v[:, :2] / v.abs().sum(1, keepdim=True)
        fold = (1 - xy.abs().flip(1)) * torch.where(xy >= 0, 1.0, -1.0)
        return torch.where(v[:, 2:] < 0, fold, xy) * 0.5 + 0.5

    x = torch.cat(feats + [octahedral(nrm), octahedral(-d)], 1)
    h = torch.cat([x, torch.zeros(n, 64 - x.shape[1], device="cuda", dtype=torch.float64)], 1)
    for layer in range(5):
        h = torch.relu(h @ W[4096 * layer:4096 * (layer + 1)].reshape(64, 64).T)
    y = h @ W[5 * 4096:5 * 4096 + 3 * 64].reshape(3, 64).T
    m = y.detach().sum(1) / 3
    loss = (((y - target) ** 2).sum(1) / (m * m + 0.01)).mean()
    loss.backward()
    return dict(loss=float(loss), weight_grads=W.grad.cpu().numpy(), table_grads=table.grad.reshape(-1).cpu().numpy(),
                predictions=y.detach().cpu().numpy())
