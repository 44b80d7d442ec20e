"""The ray-tracing library's performance cases.

Each case is a call, or the short sequence of calls, that a program built on
the library makes through ``atlas_rt``: ray queries from a thousand rays (a
picking or audio query of a game frame) to a million, the camera pass of a
renderer, batched and instanced scenes, the double-precision re-test, the
path tracer on an opaque and on an alpha-tested scene, the screen-space and
probe passes, and the radiance cache's inference and training gradients.

Scenes and sizes are the repository's own workloads (``atlas_rt.scenes``,
``atlas_rt.ptscene``) or generic ones of the same kind.  Buffers are device
memory and calls go to the default stream, with the default context
configuration, unless the case says otherwise.  Hit records hold integers
beside floats (triangle and instance index, flags) and are returned through
a 32-bit integer view of the whole buffer: the traversal promises the
shader's results bit for bit.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "atlas-engine_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import atlas_rt  # noqa: E402
from atlas_rt import BVH, MASK_ALL, MASK_SHADOW, gbuffer, ptscene, scenes  # noqa: E402

F32 = np.float32
INF = 1e12


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # A game frame's few rays (picking, line of sight, audio): latency.
        {"name": "closest_small", "kind": "trace", "any": False, "tris": 4096, "rays": 1000},
        # The plain ray cast over 65,536 random triangles, closest hits.
        {"name": "closest_random", "kind": "trace", "any": False, "tris": 65536, "rays": 1 << 20},
        # Occlusion of an odd number of incoherent rays on a larger mesh.
        {"name": "any_random", "kind": "trace", "any": True, "tris": 262144, "rays": 300007},
        # One camera pass of the terrain + boxes scene: primary hits, bounce and
        # shadow spawn, bounce hits, shadow occlusion, resolved to pixels.
        {"name": "camera_pass", "kind": "camera", "grid": 512, "boxes": 200, "width": 1920, "height": 1080},
        # 64 meshes of uneven size with uneven ray batches, half of them closest
        # hits, half occlusion, replayed from a plan.
        {"name": "batched_64", "kind": "batched", "meshes": 64, "tris": 100000, "rays": 262144},
        # A two-level scene of many instances: closest hits and masked shadow rays.
        {"name": "scene_instances", "kind": "scene", "instances": 512, "tris": 20000, "rays": 400009},
        # Closest hits with the double-precision re-test of their near ties, for a
        # consumer that needs the exact nearest triangle; odd resolution.
        {"name": "near_ties", "kind": "retest", "grid": 512, "boxes": 200, "width": 961, "height": 541},
        # A progressive path tracer's sample at full resolution, opaque scene.
        {"name": "pathtrace_hd", "kind": "pathtrace", "grid": 512, "boxes": 200, "width": 1920, "height": 1080,
         "spp": 1, "bounces": 3},
        # A real-time frame at a small, odd resolution of a scene with alpha-tested
        # and partially opaque surfaces, with the temporal pass's G-buffer.
        {"name": "realtime_foliage", "kind": "realtime", "grid": 128, "boxes": 400, "width": 321, "height": 181,
         "bounces": 3},
        # The renderer's indirect-light passes of one frame: ambient occlusion,
        # reflections, diffuse GI and the DDGI probe rays.
        {"name": "gi_passes", "kind": "passes", "grid": 512, "boxes": 200, "width": 1280, "height": 720,
         "probes": 1000, "probe_rays": 144},
        # Radiance-cache queries of a frame.
        {"name": "cache_predict", "kind": "predict", "records": 500001, "log2_table": 19},
        # Gradients of one training batch (65,536 records) of the radiance cache.
        {"name": "cache_gradients", "kind": "gradients", "records": 65536, "log2_table": 19},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "camera", "batched", "scene", "retest", "pathtrace", "realtime", "passes",
                       "predict", "gradients"])
    # an image of _log-uniform area and an aspect ratio between 1:1 and 2:1
    def image(lo, hi):
        area, aspect = _log(rng, lo, hi), rng.uniform(1.0, 2.0)
        w = max(8, int(round(math.sqrt(area * aspect))))
        return {"width": w, "height": max(8, area // w)}

    ground = {"grid": _log(rng, 64, 512), "boxes": _log(rng, 10, 200)}
    if kind == "trace":
        return {"kind": kind, "any": rng.random() < 0.5, "tris": _log(rng, 1000, 300000),
                "rays": _log(rng, 500, 1 << 20)}
    if kind == "camera":
        return {"kind": kind, **ground, **image(20000, 1920 * 1080)}
    if kind == "batched":
        return {"kind": kind, "meshes": _log(rng, 2, 64), "tris": _log(rng, 4000, 100000),
                "rays": _log(rng, 8192, 262144)}
    if kind == "scene":
        return {"kind": kind, "instances": _log(rng, 2, 512), "tris": _log(rng, 1000, 20000),
                "rays": _log(rng, 1000, 400000)}
    if kind == "retest":
        return {"kind": kind, **ground, **image(10000, 961 * 541)}
    if kind == "pathtrace":
        return {"kind": kind, **ground, **image(20000, 1920 * 1080), "spp": 1, "bounces": rng.randint(1, 3)}
    if kind == "realtime":
        return {"kind": kind, "grid": _log(rng, 32, 128), "boxes": _log(rng, 20, 400), **image(10000, 640 * 360),
                "bounces": rng.randint(1, 3)}
    if kind == "passes":
        return {"kind": kind, **ground, **image(20000, 1280 * 720), "probes": _log(rng, 50, 1000),
                "probe_rays": _log(rng, 32, 144)}
    return {"kind": kind, "records": _log(rng, 1000, 500000 if kind == "predict" else 65536),
            "log2_table": rng.randint(14, 19)}


def _trace_work(rays, tris, out_bytes):
    """A ray reads its 48-byte record, writes its result and descends about one
    root-to-leaf path: two box tests (48 operations) per level, two triangle
    tests (60 each).  The hierarchy (one 64-byte node and one 48-byte triangle
    per triangle) is read once, or less when few rays touch it."""
    levels = math.log2(max(2, tris)) + 1
    return {"bytes": rays * (48 + out_bytes) + min(112 * tris, int(112 * levels * rays)),
            "flops": int(rays * (48 * levels + 120))}


def _sum(*parts):
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


def work(case):
    kind = case["kind"]
    if kind == "trace":
        return _trace_work(case["rays"], case["tris"], 1 if case["any"] else 32)
    if kind == "batched":
        sizes = _batch_sizes(case)
        return _sum(*[_trace_work(s["n_rays"], s["n_tris"], 1 if s["any"] else 32) for s in sizes])
    if kind == "scene":
        n, t = case["rays"], case["tris"]
        one = _trace_work(n, t * case["instances"], 32)
        meshes = 3 * 112 * t + 64 * case["instances"]
        return {"bytes": n * (48 + 32 + 48 + 1) + meshes, "flops": 2 * one["flops"]}
    if kind in ("predict", "gradients"):
        n, params = case["records"], 5 * 64 * 64 + 16 * 64
        table = 16 * 2 ** case["log2_table"]
        touched = min(table * 4, n * 16 * 8 * 4)
        if kind == "predict":
            return {"bytes": n * (64 + 16) + touched + 2 * params, "flops": 2 * n * params}
        # the whole gradient is an output
        return {"bytes": n * 64 + touched + 2 * params + 8 * table + 4 * params, "flops": 6 * n * params}
    n = case["width"] * case["height"]
    tris = 2 * case["grid"] ** 2 + 12 * case["boxes"]
    if kind == "retest":
        one = _trace_work(n, tris, 32)
        return {"bytes": one["bytes"] + 32 * n, "flops": one["flops"]}
    if kind == "camera":
        # primary hits of every pixel, bounce hits and shadow occlusion of about half of them
        one = _trace_work(n, tris, 32)
        return {"bytes": 2 * 32 * n + n + 112 * tris, "flops": 2 * one["flops"]}
    if kind in ("pathtrace", "realtime"):
        # per sample about two closest hits and two shadow rays per pixel
        one = _trace_work(n, tris, 32)
        return {"bytes": 16 * n + 208 * tris, "flops": 4 * one["flops"]}
    # passes: per pixel an occlusion ray, a reflected and a GI ray with a shadow ray each
    probes = case["probes"] * case["probe_rays"]
    one = _trace_work(n + probes, tris, 32)
    return {"bytes": n * (3 * 12 + 36) + 16 * probes + 208 * tris, "flops": 4 * one["flops"]}


# ---------------------------------------------------------------------------
# Preparation
# ---------------------------------------------------------------------------

def _upload(ctx, tris):
    bvh = BVH(tris)
    return ctx.upload_mesh(bvh.nodes, bvh.pack_triangles())


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _prepare_trace(case, seed):
    ctx = atlas_rt.Context()
    mesh = _upload(ctx, scenes.random_triangles(case["tris"], seed=seed))
    rays = _cuda(scenes.pack_rays(*scenes.sphere_rays(case["rays"], seed=seed + 1)))
    n = case["rays"]
    out = torch.zeros(n, dtype=torch.uint8, device="cuda") if case["any"] else torch.zeros((n, 8), device="cuda")
    return {"ctx": ctx, "mesh": mesh, "rays": rays, "out": out}


def _camera(case, seed):
    """The default view of the terrain, moved a little with the seed."""
    r = np.random.default_rng(seed)
    eye = (50.0 + r.uniform(-8, 8), 45.0 + r.uniform(-4, 4), -22.0 + r.uniform(-4, 4))
    return scenes.pinhole_camera(case["width"], case["height"], eye=eye)


def _prepare_camera(case, seed):
    ctx = atlas_rt.Context()
    tris, _ = scenes.terrain_boxes(seed=seed, grid=case["grid"], n_boxes=case["boxes"])
    n = case["width"] * case["height"]
    # queues whose unused slots name places past the image's pixels
    queues = []
    for _ in range(2):
        q = torch.zeros((n, 12), device="cuda")
        q.view(torch.int32)[:, 3] = torch.arange(n, 2 * n, dtype=torch.int32, device="cuda")
        queues.append(q)
    return {"ctx": ctx, "mesh": _upload(ctx, tris), "cam": atlas_rt.make_camera(_camera(case, seed)), "n": n,
            "params": atlas_rt.make_bounce_params(seed=seed), "hits": torch.zeros((n, 8), device="cuda"),
            "secondary": queues[0], "shadow": queues[1], "counts": torch.zeros(2, dtype=torch.int32, device="cuda"),
            "secondary_hits": torch.zeros((n, 8), device="cuda"),
            "occluded": torch.zeros(n, dtype=torch.uint8, device="cuda"),
            "bounce": torch.zeros((2 * n, 8), dtype=torch.int32, device="cuda"),
            "shade": torch.zeros(2 * n, dtype=torch.uint8, device="cuda")}


def _run_camera(s):
    ctx, n = s["ctx"], s["n"]
    ctx.trace_camera_closest(s["mesh"], s["cam"], s["hits"], 0.0, INF)
    s["counts"].zero_()
    ctx.spawn_bounce_camera(s["mesh"], s["cam"], s["hits"], s["params"], s["secondary"], s["shadow"], s["counts"])
    ctx.trace_closest_queue(s["mesh"], s["secondary"], s["counts"], n, 0.0, INF, s["secondary_hits"])
    ctx.trace_any_queue(s["mesh"], s["shadow"], s["counts"][1:], n, 0.0, INF - 0.2, s["occluded"])
    # the queues are in no particular order: results go to their pixels by ray ID
    s["bounce"].index_copy_(0, s["secondary"].view(torch.int32)[:, 3].long(), s["secondary_hits"].view(torch.int32))
    s["shade"].index_copy_(0, s["shadow"].view(torch.int32)[:, 3].long(), s["occluded"])
    return {"primary": s["hits"].view(torch.int32), "counts": s["counts"], "bounce": s["bounce"][:n],
            "shadow": s["shade"][:n]}


def _batch_sizes(case):
    """Triangle and ray counts, log-uniform and the same for every seed."""
    return scenes.batched_scenes(case["meshes"], tri_range=(1000, case["tris"]), ray_range=(4096, case["rays"]))


def _prepare_batched(case, seed):
    ctx = atlas_rt.Context()
    sizes = _batch_sizes(case)
    n_hit = sum(z["n_rays"] for z in sizes if not z["any"])
    n_any = sum(z["n_rays"] for z in sizes if z["any"])
    hits = torch.zeros((n_hit, 8), device="cuda")
    occ = torch.zeros(n_any, dtype=torch.uint8, device="cuda")
    rays, batches, at = [], [], [0, 0]
    for i, z in enumerate(sizes):
        r = _cuda(scenes.pack_rays(*scenes.sphere_rays(z["n_rays"], seed=seed + 2 * i + 1)))
        rays.append(r)
        k = 1 if z["any"] else 0
        out = (occ if z["any"] else hits)[at[k]:at[k] + z["n_rays"]]
        at[k] += z["n_rays"]
        batches.append({"mesh": _upload(ctx, scenes.random_triangles(z["n_tris"], seed=seed + 2 * i)), "any": z["any"],
                        "rays": r, "out": out, "n_rays": z["n_rays"], "tmin": 1e-4, "tmax": 10.0})
    return {"ctx": ctx, "rays": rays, "hits": hits, "occ": occ, "plan": ctx.batch_plan(batches)}


def _prepare_scene(case, seed):
    ctx = atlas_rt.Context()
    r = np.random.default_rng(seed)
    bvhs = [BVH(scenes.random_triangles(case["tris"], seed=seed + k)) for k in range(3)]
    ids = [ctx.upload_mesh(b.nodes, b.pack_triangles()) for b in bvhs]
    bounds = [atlas_rt.mesh_bounds(b) for b in bvhs]
    instances, boxes = [], []
    for i in range(case["instances"]):
        q = np.linalg.qr(r.normal(size=(3, 3)))[0]
        model = np.eye(4)
        model[:3, :3] = q * r.uniform(3.0, 9.0)
        model[:3, 3] = r.uniform(0.0, 100.0, 3)
        k = i % 3
        # about a third of the instances cast no shadow
        instances.append(atlas_rt.make_instance(model, ids[k], MASK_ALL | (MASK_SHADOW if r.random() < 0.66 else 0)))
        boxes.append(atlas_rt.transform_aabb(*bounds[k], model))
    ctx.scene_build(np.array(instances), np.array(boxes))
    n = case["rays"]
    o, d = scenes.sphere_rays(n, seed=seed + 7)
    rays = _cuda(scenes.pack_rays((o * F32(100.0)).astype(F32), d))
    so = r.uniform(0.0, 100.0, (n, 3)).astype(F32)
    sd = scenes.sphere_rays(n, seed=seed + 8)[1]
    return {"ctx": ctx, "rays": rays, "shadow": _cuda(scenes.pack_rays(so, sd)),
            "hits": torch.zeros((n, 8), device="cuda"), "occ": torch.zeros(n, dtype=torch.uint8, device="cuda")}


def _prepare_retest(case, seed):
    ctx = atlas_rt.Context()
    tris, _ = scenes.terrain_boxes(seed=seed, grid=case["grid"], n_boxes=case["boxes"])
    n = case["width"] * case["height"]
    rays = torch.zeros((n, 12), device="cuda")
    ctx.raygen(atlas_rt.make_camera(_camera(case, seed)), rays)
    return {"ctx": ctx, "mesh": _upload(ctx, tris), "rays": rays, "hits": torch.zeros((n, 8), device="cuda"),
            "out": torch.zeros((n, 8), device="cuda")}


def _prepare_pathtrace(case, seed):
    ctx = atlas_rt.Context()
    ptscene.upload(ctx, ptscene.build(seed=seed, grid=case["grid"], n_boxes=case["boxes"]))
    n = case["width"] * case["height"]
    return {"ctx": ctx, "cam": atlas_rt.make_camera(_camera(case, seed)), "spp": case["spp"], "seed": seed & 0xFFFF,
            "bounces": case["bounces"], "accum": torch.zeros((n, 4), device="cuda")}


def _prepare_realtime(case, seed):
    """Terrain with boxes, of which a third is cut out by an opacity texture
    (foliage cards, fences) and a sixth half transparent."""
    ctx = atlas_rt.Context()
    r = np.random.default_rng(seed)
    sc = ptscene.build(seed=seed, grid=case["grid"], n_boxes=case["boxes"])
    bvh, obj = sc["bvh"], sc["obj"]
    by_object = r.choice([-1.0, -1.0, 0.5, 1.0, 1.0, 1.0], size=int(obj.max()) + 1)
    by_object[0] = by_object[sc["light_obj"]] = 1.0
    opacity = by_object[obj].astype(F32)
    shading = bvh.pack_shading(sc["normals"], obj, opacity)
    bvh.pack_attributes(shading, (sc["tris"][:, :, [0, 2]] * F32(0.25)).reshape(-1, 6), sc["normals"])
    mesh = ctx.upload_mesh(bvh.nodes, bvh.pack_triangles(obj, opacity), shading)
    ctx.scene_build(np.array([atlas_rt.make_instance(np.eye(4), mesh, MASK_ALL | MASK_SHADOW)]),
                    np.concatenate(atlas_rt.mesh_bounds(bvh))[None, :])
    mats = sc["materials"]
    mats["opacityTexture"][by_object < 0] = 0
    mats["opacity"][by_object == 0.5] = 0.5
    ctx.set_materials(mats)
    ctx.set_textures([np.where(r.random((256, 256)) < 0.5, 0, 255).astype(np.uint8)])
    ctx.set_lights(ptscene.lights_for(sc, shading))
    w, h = case["width"], case["height"]
    camd = _camera(case, seed)
    eye = camd["location"].astype(np.float64)
    view = gbuffer.look_at(eye, (50.0, 0.0, 48.0))
    proj = gbuffer.perspective(60.0, w / h, 0.5, 400.0)
    last = proj @ gbuffer.look_at(eye + (0.2, 0.0, 0.1), (50.0, 0.0, 48.0))
    planes = {"depth": torch.zeros((h, w), device="cuda"),
              "material_idx": torch.zeros((h, w), dtype=torch.int32, device="cuda"),
              "normal": torch.zeros((h, w, 2), device="cuda"), "velocity": torch.zeros((h, w, 2), device="cuda"),
              "view": view, "proj": proj, "pv_last": last}
    return {"ctx": ctx, "cam": atlas_rt.make_camera(camd), "bounces": case["bounces"], "seed": seed & 0xFFFF,
            "frame": torch.zeros((3, h, w), dtype=torch.int32, device="cuda"), "planes": planes}


def _run_realtime(s):
    s["ctx"].pathtrace_realtime(s["cam"], s["frame"], max_radiance=20.0, spp=1, max_bounces=s["bounces"],
                                seed=s["seed"], gbuffer=s["planes"])
    # at one sample per pixel the frame holds the radiance's float bits
    return {"frame": s["frame"].view(torch.float32),
            **{k: s["planes"][k] for k in ("depth", "material_idx", "normal", "velocity")}}


def _prepare_passes(case, seed):
    ctx = atlas_rt.Context()
    r = np.random.default_rng(seed)
    sc = ptscene.build(seed=seed, grid=case["grid"], n_boxes=case["boxes"])
    _, shading, _, _ = ptscene.upload(ctx, sc)
    w, h = case["width"], case["height"]
    view = gbuffer.look_at(_camera(case, seed)["location"], (50.0, 0.0, 50.0))
    gb = gbuffer.device_gbuffer(ctx, shading, view, gbuffer.perspective(60.0, w / h, 0.5, 400.0), w, h)
    gb["roughness"] = _cuda(r.uniform(0.0, 1.0, (h, w)).astype(F32))
    probes = np.zeros((case["probes"], 4), F32)
    probes[:, 0:3] = r.uniform((0.0, 2.0, 0.0), (100.0, 40.0, 100.0), (case["probes"], 3))
    probes[:, 3] = np.where(r.random(case["probes"]) < 0.2, 2, 1).astype(np.int32).view(F32)
    dirs = np.zeros((case["probe_rays"], 4), F32)
    dirs[:, 0:3] = scenes.sphere_rays(case["probe_rays"], seed=seed + 3)[1]
    rot = np.eye(4)
    rot[:3, :3] = np.linalg.qr(r.normal(size=(3, 3)))[0]
    return {"ctx": ctx, "gb": gb, "seed": seed & 0xFFFF, "probes": _cuda(probes), "dirs": _cuda(dirs), "rot": rot,
            "ao": torch.zeros((h, w), device="cuda"), "reflections": torch.zeros((h, w, 4), device="cuda"),
            "gi": torch.zeros((h, w, 4), device="cuda"),
            "probe_hits": torch.zeros((case["probes"] * case["probe_rays"], 4), device="cuda")}


def _run_passes(s):
    ctx, gb, seed = s["ctx"], s["gb"], s["seed"]
    ctx.rtao(gb, s["ao"], radius=10.0, frame_seed=seed)
    ctx.reflections(gb, s["reflections"], roughness_cutoff=0.9, frame_seed=seed)
    ctx.rtgi(gb, s["gi"], frame_seed=seed)
    ctx.ddgi_trace(s["probes"], s["dirs"], s["rot"], s["probe_hits"], ray_dirs_inactive=s["dirs"],
                   inactive_ray_count=s["dirs"].shape[0] // 4, frame_seed=seed)
    # probe hits are packed half pairs
    return {"ao": s["ao"], "reflections": s["reflections"], "gi": s["gi"],
            "probe_hits": s["probe_hits"].view(torch.int32)}


# ---- radiance cache: records and parameters, made from the seed alone ----

_LO, _HI = (0.0, -2.0, 0.0), (100.0, 62.0, 100.0)


def _cache_inputs(case, seed):
    """Records on a terrain-like surface (queries come from visible surfaces in
    image order, so neighbours lie close), and parameters that the cache's
    BF16 weights and FP16 table hold without rounding."""
    r = np.random.default_rng(seed)
    n = case["records"]
    side = math.ceil(math.sqrt(n))
    i = np.arange(n)
    x, z = (i % side + r.random(n)) / side * 100.0, (i // side + r.random(n)) / side * 100.0
    rec = np.zeros((n, 16), F32)
    rec[:, 0], rec[:, 2] = x, z
    rec[:, 1] = 8.0 * np.sin(x * 0.11) * np.cos(z * 0.07) + 10.0
    rec[:, 3] = r.uniform(0.05, 1.0, n)
    d, nn = r.normal(size=(n, 3)), r.normal(size=(n, 3)) * 0.3 + (0.0, 1.0, 0.0)
    rec[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rec[:, 8:11] = nn / np.linalg.norm(nn, axis=1, keepdims=True)
    rec[:, 11] = r.integers(0, 3, n)
    rec[:, 12:15] = r.uniform(0.0, 0.5, (n, 3))
    rec[:, 15] = 1.0
    mlp = torch.from_numpy((r.normal(size=5 * 64 * 64 + 16 * 64) * 0.18).astype(F32)).bfloat16().float().numpy()
    grid = (r.random(16 * 2 ** case["log2_table"] * 2, dtype=F32) - F32(0.5)).astype(np.float16).astype(F32)
    return rec, mlp, grid


def _prepare_cache(case, seed):
    rec, mlp, grid = _cache_inputs(case, seed)
    ctx = atlas_rt.Context()
    rc = atlas_rt.RadianceCache(ctx, _LO, _HI, log2_table=case["log2_table"], seed=seed & 0xFFFF)
    rc.set_params(mlp, grid)
    s = {"ctx": ctx, "rc": rc, "records": _cuda(rec)}
    if case["kind"] == "predict":
        s["out"] = torch.zeros((case["records"], 4), device="cuda")
    else:
        s["grad_mlp"] = torch.zeros(rc.n_mlp, device="cuda")
        s["grad_grid"] = torch.zeros(rc.n_grid, device="cuda")
    return s


def prepare(case, seed):
    kind = case["kind"]
    make = {"trace": _prepare_trace, "camera": _prepare_camera, "batched": _prepare_batched, "scene": _prepare_scene,
            "retest": _prepare_retest, "pathtrace": _prepare_pathtrace, "realtime": _prepare_realtime,
            "passes": _prepare_passes, "predict": _prepare_cache, "gradients": _prepare_cache}
    return {"kind": kind, "any": case.get("any", False), **make[kind](case, seed)}


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "trace":
        if s["any"]:
            return ctx.trace_any(s["mesh"], s["rays"], 1e-4, 10.0, out=s["out"])
        return ctx.trace_closest(s["mesh"], s["rays"], 1e-4, 10.0, out=s["out"]).view(torch.int32)
    if kind == "camera":
        return _run_camera(s)
    if kind == "batched":
        s["plan"].launch()
        return {"hits": s["hits"].view(torch.int32), "occluded": s["occ"]}
    if kind == "scene":
        ctx.trace_scene_closest(s["rays"], 0.0, INF, out=s["hits"])
        ctx.trace_scene_any(s["shadow"], 0.0, 40.0, cull_mask=MASK_SHADOW, out=s["occ"])
        return {"hits": s["hits"].view(torch.int32), "occluded": s["occ"]}
    if kind == "retest":
        ctx.trace_closest(s["mesh"], s["rays"], 0.0, INF, out=s["hits"])
        ctx.retest_near_ties(s["mesh"], s["rays"], s["hits"], 0.0, INF, s["out"], count=False)
        return {"hits": s["hits"].view(torch.int32), "exact_hits": s["out"].view(torch.int32)}
    if kind == "pathtrace":
        s["accum"].zero_()
        ctx.pathtrace(s["cam"], s["accum"], spp=s["spp"], max_bounces=s["bounces"], seed=s["seed"])
        return s["accum"]
    if kind == "realtime":
        return _run_realtime(s)
    if kind == "passes":
        return _run_passes(s)
    if kind == "predict":
        s["rc"].predict(s["records"], s["out"])
        return s["out"]
    loss = s["rc"].gradients(s["records"], s["grad_mlp"], s["grad_grid"])
    return {"loss": loss, "mlp": s["grad_mlp"], "grid": s["grad_grid"]}


# ---------------------------------------------------------------------------
# Exact results of the radiance cache in 64 bits (the traversal's outputs are
# bit patterns, the images Monte Carlo estimates)
# ---------------------------------------------------------------------------

def _corners(pos, level, T):
    """Table index and weight of the 8 corners of each position's cell."""
    growth = math.exp((math.log(2048) - math.log(16)) / 15)
    res = math.floor(16 * growth ** level + 1e-6)
    stride = res + 1
    lo = torch.tensor(_LO, dtype=torch.float32, device=pos.device)
    scale = 1.0 / (torch.tensor(_HI, dtype=torch.float32, device=pos.device) - lo)
    # the cell is found in 32 bits, as the method defines it
    p = ((pos - lo) * scale).clamp(0.0, 0.999999) * float(res)
    cell = torch.floor(p)
    f = (p - cell).double()
    cell = cell.long()
    for k in range(8):
        bits = (k & 1, (k >> 1) & 1, k >> 2)
        c = [cell[:, a] + bits[a] for a in range(3)]
        w = torch.ones_like(f[:, 0])
        for a in range(3):
            w = w * (f[:, a] if bits[a] else 1.0 - f[:, a])
        if stride ** 3 <= T:
            i = c[0] + c[1] * stride + c[2] * stride * stride
        else:
            i = (c[0] ^ (c[1] * 2654435761 & 0xFFFFFFFF) ^ (c[2] * 805459861 & 0xFFFFFFFF)) & (T - 1)
        yield i, w


def _harmonics(d):
    x, y, z = d[:, 0], d[:, 1], d[:, 2]
    xx, yy, zz = x * x, y * y, z * z
    return torch.stack([
        torch.full_like(x, 0.28209479177387814), -0.48860251190291987 * y, 0.48860251190291987 * z,
        -0.48860251190291987 * x, 1.0925484305920792 * x * y, -1.0925484305920792 * y * z,
        0.94617469575756008 * zz - 0.31539156525252005, -1.0925484305920792 * x * z,
        0.54627421529603959 * (xx - yy), 0.59004358992664352 * y * (yy - 3.0 * xx), 2.8906114426405538 * x * y * z,
        0.45704579946446572 * y * (1.0 - 5.0 * zz), 0.3731763325901154 * z * (5.0 * zz - 3.0),
        0.45704579946446572 * x * (1.0 - 5.0 * zz), 1.4453057213202769 * z * (xx - yy),
        0.59004358992664352 * x * (3.0 * yy - xx)], 1)


def exact(case, seed):
    if case["kind"] not in ("predict", "gradients"):
        return None
    rec, mlp, grid = _cache_inputs(case, seed)
    T = 2 ** case["log2_table"]
    rec = torch.from_numpy(rec).cuda()
    mlp = torch.from_numpy(mlp).cuda().double()
    table = torch.from_numpy(grid).cuda().double().reshape(16, T, 2)
    hidden = [mlp[k * 4096:(k + 1) * 4096].reshape(64, 64) for k in range(5)]
    last = mlp[5 * 4096:].reshape(16, 64)
    n = len(rec)
    grads = case["kind"] == "gradients"
    out = torch.zeros((n, 4), dtype=torch.float64, device="cuda")
    g_hidden = [torch.zeros_like(w) for w in hidden]
    g_last, g_table = torch.zeros_like(last), torch.zeros_like(table) if grads else None
    loss = 0.0
    for a in range(0, n, 65536):
        q = rec[a:a + 65536]
        X = torch.zeros((len(q), 64), dtype=torch.float64, device="cuda")
        for level in range(16):
            for i, w in _corners(q[:, 0:3], level, T):
                X[:, 2 * level:2 * level + 2] += w[:, None] * table[level, i]
        X[:, 32:48] = _harmonics(q[:, 4:7].double())
        X[:, 48:51], X[:, 51], X[:, 52] = q[:, 8:11].double(), q[:, 3].double(), q[:, 11].double()
        acts = [X]
        for w in hidden:
            acts.append((acts[-1] @ w.T).clamp(min=0.0))
        p = (acts[-1] @ last.T)[:, :3]
        out[a:a + 65536, :3] = p
        if not grads:
            continue
        t = q[:, 12:15].double()
        den = p * p + 0.01
        loss += float(((p - t) ** 2 / den).sum()) / (3 * n)
        dp = torch.zeros((len(q), 16), dtype=torch.float64, device="cuda")
        dp[:, :3] = 2.0 * (p - t) / den / (3 * n)
        g_last += dp.T @ acts[5]
        d = dp @ last
        for k in range(4, -1, -1):
            d = d * (acts[k + 1] > 0)
            g_hidden[k] += d.T @ acts[k]
            d = d @ hidden[k]
        for level in range(16):
            for i, w in _corners(q[:, 0:3], level, T):
                g_table[level].index_add_(0, i, w[:, None] * d[:, 2 * level:2 * level + 2])
    if not grads:
        return out
    return {"loss": loss, "mlp": torch.cat([g.reshape(-1) for g in g_hidden] + [g_last.reshape(-1)]),
            "grid": g_table.reshape(-1)}
