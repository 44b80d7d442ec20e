"""The traversal's launch forms: stack variants chosen by tree depth, and
launches of few rays, which fill only some lanes of each warp.  Every form
returns the same bits: the oracle's nearest triangle for the stacks, the
records of a full launch for the first rays of a small one."""
import ctypes as C

import numpy as np
import pytest

import atlas_rt
import pyoracle
from atlas_rt import BVH, _native, scenes
from test_trace_gpu import chain_bvh, packed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entries", [30, 31, 32, 33, 126, 127, 128, 129])
def test_stack_variants_at_their_edges(ctx, entries):
    """A chain that needs exactly this many stack entries, around the shared
    memory alone (31 and the end marker), the usual 128 and the deep stack."""
    nodes, tris = chain_bvh(entries + 1)
    mid = ctx.upload_mesh(nodes, tris)
    rays8 = scenes.rays8(np.tile(np.array([[0.5, 0.5, -1.0]], np.float32), (70, 1)),
                         np.tile(np.array([[0.01, -0.02, 1.0]], np.float32), (70, 1)), 0.0, 1e4)
    hits = ctx.trace_closest(mid, packed(rays8), 0.0, 1e4)
    ptr, tuv = pyoracle.closest_glsl(nodes.view(np.float32).reshape(-1, 16), tris, rays8)
    assert np.array_equal(hits["triPtr"], ptr) and (ptr == entries).all()
    assert np.array_equal(hits["t"].view(np.uint32), tuv[:, 0].view(np.uint32))
    assert (hits["flags"] & 0xC == 0).all()
    assert ctx.trace_any(mid, packed(rays8), 0.0, 1e4).all()


@pytest.fixture(scope="module")
def few():
    """A mesh, a two-instance scene of it, 60,000 rays and their full-launch results."""
    import torch
    c = atlas_rt.Context(device=0)
    b = BVH(scenes.random_triangles(9000, seed=11))
    gt = b.pack_triangles()
    mid = c.upload_mesh(b.nodes, gt)
    lo, hi = atlas_rt.mesh_bounds(b)
    models = [np.eye(4), np.diag([1.5, 0.7, 1.1, 1.0])]
    c.scene_build(np.array([atlas_rt.make_instance(m, mid, atlas_rt.MASK_ALL) for m in models]),
                  np.array([atlas_rt.transform_aabb(lo, hi, m) for m in models]))
    rays = torch.from_numpy(scenes.pack_rays(*scenes.sphere_rays(60000, seed=12))).cuda()
    d = {"ctx": c, "mid": mid, "rays": rays, "torch": torch, "bvh": b, "gt": gt}
    d["full"] = {k: run(d, k, len(rays)) for k in ("closest", "any", "scene", "queue", "noalloc")}
    yield d
    c.close()


def run(d, kind, n):
    c, rays, torch = d["ctx"], d["rays"], d["torch"]
    hits = torch.full((len(rays), 8), float("nan"), device="cuda")
    occ = torch.full((len(rays),), 7, dtype=torch.uint8, device="cuda")
    if kind == "closest":
        c.trace_closest(d["mid"], rays, 1e-4, 10.0, out=hits, n_rays=n)
    elif kind == "any":
        c.trace_any(d["mid"], rays, 1e-4, 10.0, out=occ, n_rays=n)
    elif kind == "scene":
        c.trace_scene_closest(rays, 1e-4, 10.0, out=hits, n_rays=n)
    elif kind == "queue":       # the count is read on the device
        c.trace_closest_queue(d["mid"], rays, torch.tensor([n], dtype=torch.int32, device="cuda"), len(rays), 1e-4,
                              10.0, hits)
    else:
        nodes, tris = torch.from_numpy(d["bvh"].nodes_f32.copy()).cuda(), torch.from_numpy(d["gt"]).cuda()
        assert _native.lib().ae_rt_trace_closest_noalloc(
            nodes.data_ptr(), len(d["bvh"].nodes), tris.data_ptr(), len(d["gt"]), rays.data_ptr(), n, C.c_float(1e-4),
            C.c_float(10.0), hits.data_ptr(), None) == 0
        torch.cuda.synchronize()
    c.synchronize()
    out = occ if kind == "any" else hits.view(torch.int32)
    return out.cpu().numpy()


# around one ray, one warp, one warp's share on every SM (8 warps of 152 SMs) and 32 lanes there
@pytest.mark.parametrize("kind", ["closest", "any", "scene", "queue", "noalloc"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 1215, 1216, 1217, 2433, 38911, 38912, 38913])
def test_few_rays_give_the_full_launch_records(few, kind, n):
    got, full = run(few, kind, n), few["full"][kind]
    untouched = np.float32("nan").view(np.int32) if kind != "any" else 7
    assert np.array_equal(got[:n], full[:n])
    assert (got[n:] == untouched).all()


@pytest.mark.parametrize("entries", [29, 30, 31, 126])
def test_transparency_stacks_on_an_opaque_chain(entries):
    """The transparency traversal of an opaque scene is the opaque one, around
    the depth where its stack leaves shared memory (one top-level entry more
    than the chain's), and for launches of one ray to several hundred."""
    nodes, tris = chain_bvh(entries + 1)
    shading = np.zeros((len(tris), 24), np.float32)
    shading[:, 0:12] = tris
    shading[:, [3, 7, 11]] = 0.0
    shading[:, 18], shading[:, 23] = 1.0, 1.0
    c = atlas_rt.Context(device=0)
    try:
        mid = c.upload_mesh(nodes, tris, shading)
        c.scene_build(np.array([atlas_rt.make_instance(np.eye(4), mid, atlas_rt.MASK_ALL)]),
                      np.array([[-1.0, -1.0, 1.0, 3.0, 3.0, entries + 1.0]], np.float32))
        rng = np.random.default_rng(entries)
        o = np.concatenate([rng.uniform(-1.5, 3.5, (700, 2)), np.full((700, 1), -1.0)], 1).astype(np.float32)
        rays = scenes.pack_rays(o, np.tile(np.array([[0.01, -0.02, 1.0]], np.float32), (700, 1)))
        want, occ = c.trace_scene_closest(rays, 0.0, 1e4), c.trace_scene_any(rays, 0.0, 1e4)
        assert 50 < (want["triPtr"] >= 0).sum() < 650
        for n in (1, 33, 700):
            got = c.trace_scene_closest_transparency(rays[:n].copy(), 0.0, 1e4)
            for k in ("t", "triPtr", "instance", "u", "v"):
                assert np.array_equal(got[k].view(np.uint32), want[k][:n].view(np.uint32)), (n, k)
            assert (got["tSecond"] == 1e4).all()
            vis = c.trace_scene_any_transparency(rays[:n].copy(), 0.0, 1e4)
            assert np.array_equal(vis, 1.0 - occ[:n].astype(np.float32))
    finally:
        c.close()


def test_retest_of_any_number_of_rays_gives_the_full_records(ctx):
    """Near-tie re-tests of one to all of 40,000 rays at mesh edges: the
    grouping of the double-precision tests does not show in the results."""
    import torch
    b = BVH(scenes.terrain_boxes(seed=5, grid=48, n_boxes=6)[0])
    mid = ctx.upload_mesh(b.nodes, b.pack_triangles())
    rng = np.random.default_rng(6)
    n = 40000
    at = b._verts.reshape(-1, 3)[rng.integers(0, 3 * b.n_input, n)]      # vertices, where triangles tie
    o = np.array([[50.0, 60.0, -20.0]], np.float32) + rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    d = (at - o).astype(np.float32)
    rays = torch.from_numpy(scenes.pack_rays(o.astype(np.float32), d / np.linalg.norm(d, axis=1, keepdims=True))).cuda()
    hits = torch.zeros((n, 8), device="cuda")
    ctx.trace_closest(mid, rays, 0.0, 1e12, out=hits)
    full = torch.zeros((n, 8), device="cuda")
    flagged = ctx.retest_near_ties(mid, rays, hits, 0.0, 1e12, full)
    assert flagged > n // 4
    for k in (1, 2, 31, 33, 1000, 2433, 20000):
        part = torch.zeros((n, 8), device="cuda")
        ctx.retest_near_ties(mid, rays, hits, 0.0, 1e12, part, n_rays=k)
        assert torch.equal(part[:k].view(torch.int32), full[:k].view(torch.int32)), k
        assert not part[k:].any()


@pytest.mark.parametrize("bounces", [1022, 1023, 1030])
def test_path_tracer_counters_past_their_sets(bounces):
    """The path tracer's per-bounce counters are used again past 1,024 bounces;
    every path has ended long before, so the image is that of 200 bounces."""
    import torch
    from atlas_rt import ptscene
    c = atlas_rt.Context(device=0)
    try:
        ptscene.upload(c, ptscene.build(seed=7, grid=16, n_boxes=4))
        cam = atlas_rt.make_camera(scenes.pinhole_camera(24, 17))
        img = []
        for b in (200, bounces):
            acc = torch.zeros((24 * 17, 4), device="cuda")
            c.pathtrace(cam, acc, spp=2, max_bounces=b)
            c.synchronize()
            img.append(acc)
        assert torch.equal(*img) and float(img[0].sum()) > 0
    finally:
        c.close()


@pytest.mark.parametrize("kinds", ["c", "a", "ac", "ca", "acca0c", "0a", "c0"])
def test_batches_of_either_kind_alone_and_mixed(few, kinds):
    """Batched launches (direct and planned) with closest-hit (c), any-hit (a)
    and empty (0) batches in any order: each gives its single launch's records."""
    torch = few["torch"]
    c, rays = few["ctx"], few["rays"]
    batches, want = [], []
    for i, k in enumerate(kinds):
        n = 0 if k == "0" else 700 * i + 33
        at = 5000 * i
        any_hit = k == "a" or (k == "0" and i % 2 == 1)
        out = torch.full((max(n, 1),), 7, dtype=torch.uint8, device="cuda") if any_hit \
            else torch.zeros((max(n, 1), 8), device="cuda")
        batches.append({"mesh": few["mid"], "any": any_hit, "rays": rays[at:], "out": out, "n_rays": n, "tmin": 1e-4,
                        "tmax": 10.0})
        want.append(few["full"]["any" if any_hit else "closest"][at:at + n])
    plan = c.batch_plan(batches)
    for launch in (lambda: c.trace_batched(batches), plan.launch, plan.launch):
        for b in batches:
            b["out"].zero_()
        launch()
        c.synchronize()
        for b, w in zip(batches, want):
            got = b["out"][:b["n_rays"]]
            got = got if b["any"] else got.view(torch.int32)
            assert np.array_equal(got.cpu().numpy().reshape(w.shape), w)
    plan.close()


@pytest.mark.parametrize("n", [1, 19455, 19456, 19457, 38912])
def test_few_rays_on_a_context_of_one_cta_per_sm(few, n):
    """With one CTA an SM configured, the grid of a small launch may not hold all
    of its rays at once (152 x 128): both sides of that line."""
    c = atlas_rt.Context(device=0, blocks_per_sm=1)
    try:
        mid = c.upload_mesh(few["bvh"].nodes, few["gt"])
        assert np.array_equal(run({**few, "ctx": c, "mid": mid}, "closest", n)[:n], few["full"]["closest"][:n])
        assert np.array_equal(run({**few, "ctx": c, "mid": mid}, "any", n)[:n], few["full"]["any"][:n])
    finally:
        c.close()


@pytest.mark.parametrize("w,h", [(353, 276), (641, 479)])
def test_path_tracer_queues_longer_than_the_shading_grid(w, h):
    """A shading block that takes several chunks of its queue gives the image
    of strips of which every block takes one; the 64-bit sums differ by the
    order of at most 20 additions."""
    import torch
    from atlas_rt import ptscene
    c = atlas_rt.Context(device=0)
    try:
        ptscene.upload(c, ptscene.build(seed=5, grid=64, n_boxes=20))
        cam = atlas_rt.make_camera(scenes.pinhole_camera(w, h))
        acc = torch.zeros((w * h, 4), device="cuda")
        img = []
        for rows in (h, 32):
            acc64 = torch.zeros((w * h, 3), device="cuda", dtype=torch.float64)
            for y in range(0, h, rows):
                c.pathtrace(cam, acc, acc64, spp=2, tile=(0, y, w, min(rows, h - y)))
            c.synchronize()
            img.append(acc64.cpu().numpy())
        np.testing.assert_allclose(img[0], img[1], rtol=20 * 2.0 ** -53, atol=0)
        assert (img[0] > 0).mean() > 0.3
    finally:
        c.close()


@pytest.mark.parametrize("cap", [1, 2, 3, 4, 5, 9, 30, 0])
@pytest.mark.parametrize("cull", [0xFFFFFFFF, 2])
def test_scene_rounds_of_several_visits_keep_the_step_cap(cap, cull):
    """Entering an instance and leaving a leaf visit the next node in the same
    round unless the burst ends there: with bursts of one step they never do,
    and every record and cap flag has to be the same."""
    import torch
    b = BVH(scenes.random_triangles(700, seed=21))
    one = np.array([[[0, 0, 0], [1, 0, 0], [0, 1, 0]]], np.float32)
    small = BVH(one.reshape(np.asarray(scenes.random_triangles(1, seed=1)).shape))
    rays = torch.from_numpy(scenes.pack_rays(*scenes.sphere_rays(30000, seed=23))).cuda()
    got = []
    for burst in (1, 2, 24):
        c = atlas_rt.Context(device=0, max_steps=cap, refill_steps=burst)
        try:
            ids = [c.upload_mesh(x.nodes, x.pack_triangles()) for x in (b, small)]
            bounds = [atlas_rt.mesh_bounds(x) for x in (b, small)]
            rng = np.random.default_rng(22)
            inst, boxes = [], []
            for i in range(24):
                model = np.eye(4)
                model[:3, :3] *= rng.uniform(0.2, 0.7)
                model[:3, 3] = rng.uniform(-1.0, 1.0, 3)
                inst.append(atlas_rt.make_instance(model, ids[i % 2], 1 + i % 3))
                boxes.append(atlas_rt.transform_aabb(*bounds[i % 2], model))
            c.scene_build(np.array(inst), np.array(boxes))
            hits = torch.zeros((len(rays), 8), device="cuda")
            occ = torch.zeros(len(rays), dtype=torch.uint8, device="cuda")
            c.trace_scene_closest(rays, 1e-4, 10.0, cull_mask=cull, out=hits)
            c.trace_scene_any(rays, 1e-4, 10.0, cull_mask=cull, out=occ)
            torch.cuda.synchronize()
            got.append((hits.cpu().numpy().view(np.uint32), occ.cpu().numpy()))
        finally:
            c.close()
    for hits, occ in got[1:]:
        assert np.array_equal(hits, got[0][0]) and np.array_equal(occ, got[0][1])
    assert (got[0][0][:, 3] & atlas_rt.HIT_FLAG_ITER_CAP).any() == (0 < cap < 30) or cap == 30


@pytest.mark.parametrize("kind", ["closest", "any", "scene", "pathtrace", "passes"])
def test_chained_launches_in_a_captured_graph(few, kind):
    """Chains of launches that are set up ahead of the previous one's end,
    recorded once and replayed twice over cleared outputs: the eager results."""
    import torch
    from atlas_rt import gbuffer, ptscene
    c = few["ctx"]
    if kind in ("pathtrace", "passes"):
        c = atlas_rt.Context(device=0)
        _, shading, _, _ = ptscene.upload(c, ptscene.build(seed=3, grid=24, n_boxes=8))
    try:
        w, h = 97, 65
        hits = torch.zeros((len(few["rays"]), 8), device="cuda")
        occ = torch.zeros(len(few["rays"]), dtype=torch.uint8, device="cuda")
        image, gi = torch.zeros((w * h, 4), device="cuda"), torch.zeros((h, w, 4), device="cuda")
        outs = [hits, occ, image, gi]
        cam = atlas_rt.make_camera(scenes.pinhole_camera(w, h))
        if kind == "passes":
            view = gbuffer.look_at((50.0, 30.0, -40.0), (50.0, 0.0, 50.0))
            gb = gbuffer.device_gbuffer(c, shading, view, gbuffer.perspective(60.0, w / h, 0.5, 400.0), w, h)

        def chain(stream):
            for _ in range(2):
                if kind == "closest":
                    c.trace_closest(few["mid"], few["rays"], 1e-4, 10.0, out=hits, stream=stream)
                elif kind == "any":
                    c.trace_any(few["mid"], few["rays"], 1e-4, 10.0, out=occ, stream=stream)
                elif kind == "scene":
                    c.trace_scene_closest(few["rays"], 1e-4, 10.0, out=hits, stream=stream)
                elif kind == "pathtrace":
                    c.pathtrace(cam, image, spp=1, stream=stream)
                else:
                    c.rtgi(gb, gi, frame_seed=5, stream=stream)

        side = torch.cuda.Stream()
        chain(side.cuda_stream)
        side.synchronize()
        want = [o.cpu().numpy().view(np.uint8).copy() for o in outs]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            for o in outs:
                o.zero_()
            chain(side.cuda_stream)
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
        for o, v in zip(outs, want):
            assert np.array_equal(o.cpu().numpy().view(np.uint8), v)
        assert any(v.any() for v in want)
    finally:
        if c is not few["ctx"]:
            c.close()


@pytest.mark.parametrize("w,h", [(17, 3), (641, 479), (1201, 701)])
def test_pass_queues_longer_than_the_shading_grid(w, h):
    """Reflections and GI of a frame whose shading blocks take several chunks
    of the queue, against the same frame with all but 96 rows at the far plane
    at a time, of whose queue every block takes one: samples are keyed by the
    pixel, so the bits are the same."""
    import torch
    from atlas_rt import gbuffer, ptscene
    c = atlas_rt.Context(device=0)
    try:
        _, shading, _, _ = ptscene.upload(c, ptscene.build(seed=9, grid=48, n_boxes=20))
        view = gbuffer.look_at((50.0, 30.0, -40.0), (50.0, 0.0, 50.0))
        gb = gbuffer.device_gbuffer(c, shading, view, gbuffer.perspective(60.0, w / h, 0.5, 400.0), w, h)
        gb["roughness"] = torch.full((h, w), 0.4, device="cuda")
        depth = gb["depth"].reshape(h, w).clone()
        full, part = torch.zeros((h, w, 4), device="cuda"), torch.zeros((h, w, 4), device="cuda")
        lit = 0.0
        for run in (c.rtgi, c.reflections):
            gb["depth"] = depth
            run(gb, full, frame_seed=5)
            for y in range(0, h, 96):
                gb["depth"] = torch.ones_like(depth)
                gb["depth"][y:y + 96] = depth[y:y + 96]
                run(gb, part, frame_seed=5)
                c.synchronize()
                assert torch.equal(part[y:y + 96].view(torch.int32), full[y:y + 96].view(torch.int32))
            lit += float(full[..., :3].sum())
        assert lit > 0
        # the largest frame's queue is longer than eight blocks of 128 an SM
        assert (int((depth < 1).sum()) > 8 * 128 * 152) == (w > 1000)
    finally:
        c.close()
