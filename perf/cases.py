"""Performance cases: the work a user of this library has it do, call by call.

Each case is one use of a public entry point over its real range of sizes; `listed`
names the ones that are tracked, `draw` gives more of the same kinds:

  camera   one frame of the camera tracing step: the lights culled to tiles and the
           primary, shadow, probe-visibility and bounce rays traced, device buffers
           (a renderer's frame) or host buffers (a caller without a GPU of its own
           kind, results copied back while the frame traces)
  rays     one batch of rays of mixed kinds against one resident scene (a physics or
           audio query, a baker's tile)
  batch    many ray buffers against many resident scenes in one launch
  serve    a burst of requests through the serving loop, host buffers in and out
  probes   an update of a light-probe field
  shade    the lighting step of a traced frame
  build    a BVH built on the GPU from a mesh

What a program keeps between calls (context, resident scene, batch, server, output
buffers) is made by `prepare`; `run` is one call as such a program makes it. A scene
is the same for every seed, as a program's scene is; cameras, rays, probe fields, sun
directions, units and colours come from the seed. All outputs are the entry points' own
words (hit records with the bits of t, masks, halves, node words): the library's
results are exact to the bit, so they are compared as whole numbers and no case has
a value in 64 bits to be near to.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from tim_raytracing_b200 import _native as N
from tim_raytracing_b200 import scenes


def listed():
    return [
        # the smallest frame: a room of 1,314 triangles at 256 x 256 with the tracing step's
        # own flags (sun, leaf lights, probe visibility); launches and latency count
        dict(name="room_256", kind="camera", scene="room", tris=1314, width=256, height=256, lights="leaf", mask=True,
             bounce=False, form="binary", host=False),
        # the benchmark frame: 100,608 triangles, 1080p, tile-culled lights and one bounce
        dict(name="frame_1080p", kind="camera", scene="field", tris=100608, width=1920, height=1080, lights="tile",
             mask=False, bounce=True, form="binary", host=False),
        # the same frame on the quantised 8-wide tree
        dict(name="frame_1080p_quantised", kind="camera", scene="field", tris=100608, width=1920, height=1080,
             lights="tile", mask=False, bounce=True, form="quantised", host=False),
        # an odd window size with the tracing step's own flags: eight short visibility segments a pixel
        dict(name="frame_odd_mask", kind="camera", scene="field", tris=100608, width=1279, height=719, lights="leaf",
             mask=True, bounce=False, form="binary", host=False),
        # the benchmark frame through host buffers: one call, culling inside, banded copies
        dict(name="frame_1080p_host", kind="camera", scene="field", tris=100608, width=1920, height=1080, lights="tile",
             mask=False, bounce=True, form="binary", host=True),
        # the smallest ray job of the serving mix, closest hits with every output
        dict(name="rays_1k", kind="rays", tris=100608, n=1000, mode="closest", full=True, form="binary"),
        # a large batch of mixed closest and occlusion rays, hit records only
        dict(name="rays_1m_mixed", kind="rays", tris=100608, n=1000003, mode="per_ray", full=False, form="binary"),
        # 16 scenes of 1K to 300K random triangles, 4K to 400K rays each, one launch
        dict(name="batch_16_scenes", kind="batch", scenes=16, max_tris=300000, max_rays=400000, form="binary"),
        # a burst of 48 requests of 1K to 64K rays over 4 scenes
        dict(name="serve_48", kind="serve", scenes=4, tris=100608, requests=48, max_rays=65536),
        # a whole probe field of 32 x 32 x 8 probes, 256 octahedral directions, 1M triangles
        dict(name="probes_1m", kind="probes", tris=999808, rx=32, ry=32, rz=8, side=16, octa=True, form="binary"),
        # the lighting step of a 1080p frame with 16 lights and a probe field
        dict(name="shade_1080p", kind="shade", tris=100608, width=1920, height=1080, lpf=12),
        # a mesh of 300K triangles, host arrays in and the tree's image out
        dict(name="build_300k", kind="build", tris=300000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["camera", "camera", "camera", "rays", "rays", "batch", "serve", "probes", "shade", "build"])
    form = rng.choice(["binary", "binary", "quantised"])
    tris = _log(rng, 2000, 300000)
    if kind == "camera":
        w = _log(rng, 64, 1920)
        h = max(16, min(1080, int(w * rng.uniform(0.5, 1.0))))
        room = rng.random() < 0.2
        return dict(kind=kind, scene="room" if room else "field", tris=1314 if room else tris, width=w, height=h,
                    lights=rng.choice(["tile", "leaf"]), mask=rng.random() < 0.5, bounce=rng.random() < 0.5, form=form,
                    host=rng.random() < 0.25)
    if kind == "rays":
        return dict(kind=kind, tris=tris, n=_log(rng, 1000, 1000000), mode=rng.choice(["closest", "any", "per_ray"]),
                    full=rng.random() < 0.5, form=form)
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(2, 16), max_tris=_log(rng, 2000, 300000),
                    max_rays=_log(rng, 8000, 400000), form=form)
    if kind == "serve":
        return dict(kind=kind, scenes=rng.randint(1, 4), tris=tris, requests=rng.randint(1, 48),
                    max_rays=_log(rng, 2000, 65536))
    if kind == "probes":
        return dict(kind=kind, tris=tris, rx=4 * rng.randint(1, 8), ry=4 * rng.randint(1, 8), rz=4 * rng.randint(1, 2),
                    side=rng.choice([8, 16]), octa=rng.random() < 0.5, form=form)
    if kind == "shade":
        w = _log(rng, 64, 1920)
        return dict(kind=kind, tris=tris, width=w, height=max(16, min(1080, int(w * rng.uniform(0.5, 1.0)))),
                    lpf=rng.randint(2, 16))
    return dict(kind=kind, tris=_log(rng, 2000, 300000))


# ---------------------------------------------------------------- scenes

@functools.lru_cache(maxsize=1)
def _sphere_mesh():
    return scenes.icosphere(3)


@functools.lru_cache(maxsize=40)
def _scene(kind, tris, seed=2):
    """The benchmark's heightfield with spheres at about `tris` triangles (one third
    field, two thirds spheres), the room, or `tris` random triangles."""
    if kind == "room":
        return scenes.room_scene()
    if kind == "random":
        return scenes.random_triangles(10000 + seed, tris)
    extent = 20.0
    grid = max(4, int(round(math.sqrt(tris / 6.0))))
    flat = scenes.heightfield_scene(seed=seed, grid=grid, n_spheres=0, extent=extent)
    v, f = _sphere_mesh()
    rng = np.random.default_rng(seed)
    k = max(0, int(round((tris - 2 * grid * grid) / len(f))))
    centre = rng.uniform((0.0, 0.0, 0.0), (extent, extent, 5.0), size=(k, 3))
    radius = np.exp(rng.uniform(math.log(0.2), math.log(1.5), size=k))
    nv, nt = flat.num_vertex, flat.num_tris
    pos = (centre[:, None] + radius[:, None, None] * v[None]).reshape(-1, 3)
    chunks = [(nv + i * len(v), len(v), nt + i * len(f), len(f)) for i in range(k)]
    return dataclasses.replace(
        flat, positions=np.concatenate([flat.positions, pos.astype(np.float32)]),
        normals=np.concatenate([flat.normals, np.tile(v, (k, 1)).astype(np.float32)]),
        chunks=np.concatenate([flat.chunks, np.array(chunks, np.uint32).reshape(-1, 4)]),
        local_idx=np.concatenate([flat.local_idx, np.tile(f, (k, 1)).astype(np.uint32)]),
        colors=np.concatenate([flat.colors, rng.uniform(0.2, 0.9, (k, 3)).astype(np.float32)]))


@functools.lru_cache(maxsize=40)
def _image(kind, tris, seed=2):
    return N.build_bvh(_scene(kind, tris, seed))


def _pinned(shape, dtype):
    t = torch.empty(shape, dtype=dtype, pin_memory=True)
    return t, t.numpy()


def _pass_data(scene, img, width, height, lpf, rng):
    """A camera near the scene's own, a little elsewhere for each seed, and its sun."""
    cam = np.array(scene.meta["cam_pos"]) + rng.uniform(-0.1, 0.1, 3)
    pd = scenes.pass_data(scene, width, height, lpf_res=(lpf, lpf, lpf), cam_pos=cam, aabb=(img.aabb[:3], img.aabb[3:]))
    sun = np.array(scene.meta["sun_dir"]) + rng.uniform(-0.1, 0.1, 3)
    pd["sunDir"] = (*(sun / np.linalg.norm(sun)), 0.0)
    return pd


@functools.lru_cache(maxsize=1)
def _stream():
    """The program's stream: device-buffer calls are ordered on it, one after another."""
    return torch.cuda.Stream().cuda_stream


def _words(*shape):
    return torch.zeros(shape, dtype=torch.int32, device="cuda")


# ---------------------------------------------------------------- camera and lighting step

def _prepare_camera(case, rng):
    scene, img = _scene(case["scene"], case["tris"]), _image(case["scene"], case["tris"])
    ctx = N.Context(0)
    wide = case["form"] == "quantised"
    sid = ctx.upload(img, scene, quant8=wide)
    w, h = case["width"], case["height"]
    flags = N.CAM_WIDE | N.CAM_PRIMARY_BINARY if wide else 0
    flags |= N.CAM_TILE_LIGHTS if case["lights"] == "tile" else 0
    flags |= (N.CAM_PROB_MASK if case["mask"] else 0) | (N.CAM_BOUNCE if case["bounce"] else 0)
    st = dict(kind="camera", host=case["host"], ctx=ctx, sid=sid, flags=flags, pd=_pass_data(scene, img, w, h, 12, rng),
              frame=int(rng.integers(1 << 20)), tx=(w + 15) // 16, ty=(h + 15) // 16)
    if case["host"]:
        st["flags"] |= N.CAM_PIPELINED | (N.CAM_DEVICE_CULL if case["lights"] == "tile" else 0)
        st["keep_out"], out = _pinned((w * h, 8), torch.int32)
        st["out"] = out.view(np.uint32)
        st["keep_bounce"], b = _pinned((w * h, 4), torch.int32)
        st["bounce"] = b.view(np.uint32) if case["bounce"] else None
    else:
        st["out"] = _words(w * h, 8)
        st["bounce"] = _words(w * h, 4) if case["bounce"] else None
        st["counts"], st["lists"] = _words(st["tx"] * st["ty"]), _words(st["tx"] * st["ty"], 16)
    return st


def _run_camera(s):
    ctx = s["ctx"]
    if s["host"]:
        ctx.trace_camera(s["sid"], s["pd"], s["flags"], s["frame"], out=s["out"], bounce_out=s["bounce"])
    else:
        tile = bool(s["flags"] & N.CAM_TILE_LIGHTS)
        if tile:
            ctx.cull_lights_dev(s["sid"], s["pd"], s["tx"], s["ty"], s["counts"], s["lists"],
                                stream=_stream())
        ctx.trace_camera_dev(s["sid"], s["pd"], s["flags"], s["frame"], s["counts"] if tile else None,
                             s["lists"] if tile else None, s["out"], s["bounce"], stream=_stream())
    return [s["out"]] + ([s["bounce"]] if s["bounce"] is not None else [])


def _prepare_shade(case, rng):
    cam = dict(scene="field", tris=case["tris"], width=case["width"], height=case["height"], lights="leaf", mask=True,
               bounce=False, form="binary", host=False)
    st = _prepare_camera(cam, rng)
    r = case["lpf"]
    st["pd"]["lpfResolution"] = (r, r, r, 0)
    _run_camera(st)
    # a field as updates leave it: a positive mean radiance and smaller directional parts
    field = rng.normal(0.0, 0.2, size=(7, r, r, r, 4))
    field[0, ..., :3] = rng.uniform(0.2, 1.5, size=(r, r, r, 3))
    field[0, ..., 3] = 0.0
    st.update(kind="shade", field=torch.from_numpy(field.astype(np.float16).view(np.int16)).cuda(),
              lit=torch.zeros((case["width"] * case["height"], 4), dtype=torch.int16, device="cuda"))
    return st


def _run_shade(s):
    L = N.lib()
    N._check(L.tim_rt_shade_camera_dev(s["ctx"].handle, s["sid"], s["pd"].ctypes.data, 0, s["out"].data_ptr(),
                                       s["field"].data_ptr(), s["lit"].data_ptr(), None, _stream()))
    return s["lit"]


# ---------------------------------------------------------------- ray batches

def _prepare_rays(case, rng):
    scene, img = _scene("field", case["tris"]), _image("field", case["tris"])
    ctx = N.Context(0)
    wide = case["form"] == "quantised"
    sid = ctx.upload(img, scene, quant8=wide)
    n = case["n"]
    mode = {"closest": N.MODE_CLOSEST, "any": N.MODE_ANY, "per_ray": N.MODE_PER_RAY}[case["mode"]]
    rays = scenes.serving_rays(int(rng.integers(1 << 30)), n, lights=scene.lights)
    return dict(kind="rays", ctx=ctx, sid=sid, n=n, mode=mode | (N.TRACE_WIDE if wide else 0),
                rays=torch.from_numpy(rays).cuda(), hit=_words(n, 4), nid=_words(n) if case["full"] else None,
                bary=_words(n, 2) if case["full"] else None)


def _run_rays(s):
    s["ctx"].trace_dev(s["sid"], s["rays"], s["n"], s["mode"], s["hit"], s["nid"], s["bary"], stream=_stream())
    return [x for x in (s["hit"], s["nid"], s["bary"]) if x is not None]


def _spread(count, lo, hi, seed):
    """`count` sizes spread over the logarithm of [lo, hi]."""
    r = np.random.default_rng(seed)
    return [int(x) for x in np.exp(r.uniform(math.log(lo), math.log(hi), count))]


def _prepare_batch(case, rng):
    ctx = N.Context(0)
    wide = case["form"] == "quantised"
    tris = _spread(case["scenes"], 1000, case["max_tris"], 3)
    rays = _spread(case["scenes"], 4000, case["max_rays"], 4)
    jobs = []
    for k, (t, n) in enumerate(zip(tris, rays)):
        sid = ctx.upload(_image("random", t, k), _scene("random", t, k), quant8=wide)
        r = torch.from_numpy(scenes.random_rays(int(rng.integers(1 << 30)), n)).cuda()
        jobs.append((sid, N.MODE_PER_RAY, n, r, _words(n, 4), None, None))
    return dict(kind="batch", ctx=ctx, jobs=jobs, batch=ctx.batch_create(jobs, wide=wide))


def _run_batch(s):
    s["ctx"].batch_launch(s["batch"], stream=_stream())
    return [j[4] for j in s["jobs"]]


def _prepare_serve(case, rng):
    ctx = N.Context(0)
    sids = [ctx.upload(_image("field", case["tris"], 2 + k), _scene("field", case["tris"], 2 + k))
            for k in range(case["scenes"])]
    sizes = _spread(case["requests"], 1000, case["max_rays"], 5)
    keep_r, rays = _pinned((sum(sizes), 8), torch.float32)
    rays[:] = scenes.serving_rays(int(rng.integers(1 << 30)), sum(sizes),
                                  lights=_scene("field", case["tris"], 2).lights)
    keep_h, hits = _pinned((sum(sizes), 4), torch.int32)
    hits[:] = 0
    first = np.concatenate([[0], np.cumsum(sizes)])
    reqs = [(sids[k % len(sids)], rays[first[k]:first[k + 1]], hits[first[k]:first[k + 1]]) for k in range(len(sizes))]
    return dict(kind="serve", ctx=ctx, server=N.Server(ctx), reqs=reqs, hits=hits, keep=(keep_r, keep_h))


def _run_serve(s):
    for sid, rays, hit in s["reqs"]:
        s["server"].submit(sid, rays, N.MODE_PER_RAY, hit)
    s["server"].drain()
    return s["hits"]


# ---------------------------------------------------------------- probes and builds

def _prepare_probes(case, rng):
    scene, img = _scene("field", case["tris"]), _image("field", case["tris"])
    ctx = N.Context(0)
    wide = case["form"] == "quantised"
    sid = ctx.upload(img, scene, quant8=wide)
    nd = case["side"] ** 2
    dirs, basis = N.probe_directions(nd, N.DIRS_OCTAHEDRAL if case["octa"] else N.DIRS_STRATIFIED, 9)
    sun = np.array([-0.4, 0.3, -1.0]) + rng.uniform(-0.1, 0.1, 3)
    res = (case["rx"], case["ry"], case["rz"])
    flags = (N.PROBE_OCTA if case["octa"] else 0) | (N.PROBE_WIDE | N.PROBE_PRIMARY_BINARY if wide else 0)
    desc = N.probe_desc(img.aabb[:3], img.aabb[3:], res, sun, (1.0, 0.95, 0.9), nd, 0.03, flags)
    field = rng.uniform(0.0, 0.5, size=(7, res[2], res[1], res[0], 4)).astype(np.float16)
    keep, sh16 = _pinned(field.shape, torch.int16)
    sh16 = sh16.view(np.uint16)
    sh16[:] = field.view(np.uint16)
    return dict(kind="probes", ctx=ctx, sid=sid, desc=desc, dirs=dirs, basis=basis, sh16=sh16, keep=keep,
                octa=case["octa"])


def _run_probes(s):
    _, _, _, octa, _ = s["ctx"].update_probes(s["sid"], s["desc"], s["dirs"], s["basis"], s["sh16"],
                                              want_octa=s["octa"])
    return [s["sh16"]] + ([octa.view(np.uint32)] if octa is not None else [])


def _prepare_build(case, rng):
    # the mesh in another unit (a power of two, so the tree keeps its shape) and repainted
    base, scale = _scene("field", case["tris"]), float(2.0 ** int(rng.integers(-3, 4)))
    lights = base.lights.copy()
    lights[:, :4] *= scale
    return dict(kind="build", ctx=N.Context(0), scene=dataclasses.replace(
        base, positions=base.positions * np.float32(scale), lights=lights,
        colors=rng.uniform(0.2, 0.9, base.colors.shape).astype(np.float32)))


def _run_build(s):
    img = N.build_bvh(s["scene"], s["ctx"], max_depth=32)
    return [img.data, img.ranges, img.aabb.view(np.uint32)]


_PREPARE = dict(camera=_prepare_camera, shade=_prepare_shade, rays=_prepare_rays, batch=_prepare_batch,
                serve=_prepare_serve, probes=_prepare_probes, build=_prepare_build)
_RUN = dict(camera=_run_camera, shade=_run_shade, rays=_run_rays, batch=_run_batch, serve=_run_serve,
            probes=_run_probes, build=_run_build)


def prepare(case, seed):
    st = _PREPARE[case["kind"]](case, np.random.default_rng(seed))
    torch.cuda.synchronize()
    return st


def run(state):
    return _RUN[state["kind"]](state)


# ---------------------------------------------------------------- the work of one pass

def _scene_bytes(tris):
    """A scene's triangles (three vertex positions' share and the record) and a tree over them."""
    return tris * (6 + 12 + 48)


def _touched_bytes(rays, tris):
    """What the rays must read of a scene: at most all of it, at least a path each."""
    return min(_scene_bytes(tris), rays * (48 * math.log2(max(2.0, tris / 4.0)) + 200))


def _ray_flops(rays, tris):
    """Two slab tests (3 x 2 subtract, 2 multiply, 4 min / max) a level of a balanced
    tree, and one leaf of four triangles (about 50 operations each)."""
    return rays * (2 * 20 * math.log2(max(2.0, tris / 4.0)) + 4 * 50)


def work(case):
    k, tris = case["kind"], case.get("tris", 0)
    if k == "camera":
        px = case["width"] * case["height"]
        second = 1 + (2 if case["lights"] == "tile" else 1) + (8 if case["mask"] else 0) + (1 if case["bounce"] else 0)
        rays = px * (1 + 0.6 * second)   # about six pixels in ten hit the scene
        return dict(bytes=_scene_bytes(tris) + px * (32 + (16 if case["bounce"] else 0)), flops=_ray_flops(rays, tris))
    if k == "shade":
        px = case["width"] * case["height"]
        # seven RGBA corners' lerps (28 channels x 7 x 3) and the lights, six pixels in ten
        return dict(bytes=px * (32 + 8) + 56 * case["lpf"] ** 3, flops=px * 0.6 * (28 * 21 + 16 * 20 + 100))
    if k == "rays":
        n = case["n"]
        return dict(bytes=_touched_bytes(n, tris) + n * (32 + 16 + (12 if case["full"] else 0)), flops=_ray_flops(n, tris))
    if k == "batch":
        t = _spread(case["scenes"], 1000, case["max_tris"], 3)
        n = _spread(case["scenes"], 4000, case["max_rays"], 4)
        return dict(bytes=sum(map(_touched_bytes, n, t)) + 48 * sum(n), flops=sum(_ray_flops(b, a) for a, b in zip(t, n)))
    if k == "serve":
        n = sum(_spread(case["requests"], 1000, case["max_rays"], 5))
        return dict(bytes=_touched_bytes(n, case["scenes"] * tris) + 48 * n, flops=_ray_flops(n, tris))
    if k == "probes":
        p = case["rx"] * case["ry"] * case["rz"]
        n = p * case["side"] ** 2
        return dict(bytes=_scene_bytes(tris) + p * (112 + (768 if case["octa"] else 0)),
                    flops=_ray_flops(3.5 * n, tris) + n * (54 + 16 * 20))
    # build: positions and records in, node and leaf words out; sorting and the treelets' costs
    return dict(bytes=tris * (6 + 12 + 80), flops=tris * 2000)
