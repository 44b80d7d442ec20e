"""Launches of one context in flight on several streams at once."""
import numpy as np
import pytest

import atlas_rt
from atlas_rt import BVH, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def meshes():
    c = atlas_rt.Context(device=0)
    b = BVH(scenes.random_triangles(9000, seed=11))
    mid = c.upload_mesh(b.nodes, b.pack_triangles())
    yield c, mid
    c.close()


def test_one_batch_table_on_two_streams(meshes):
    """Two launches of the same batches, the second issued while the first
    runs: each hands out all of its rays, whatever the other has taken."""
    import torch
    c, mid = meshes
    n = 400_000
    rays = torch.from_numpy(scenes.pack_rays(*scenes.sphere_rays(n, seed=12))).cuda()
    hits, occ = torch.zeros((n, 8), device="cuda"), torch.zeros(n, dtype=torch.uint8, device="cuda")
    batches = [{"mesh": mid, "any": False, "rays": rays, "out": hits, "n_rays": n, "tmin": 1e-4, "tmax": 10.0},
               {"mesh": mid, "any": True, "rays": rays, "out": occ, "n_rays": n, "tmin": 1e-4, "tmax": 10.0}]
    c.trace_batched(batches)
    c.synchronize()
    want = hits.clone(), occ.clone()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(10):
        hits.zero_()
        occ.zero_()
        torch.cuda.synchronize()
        for s in streams:
            c.trace_batched(batches, stream=s.cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(hits.view(torch.int32), want[0].view(torch.int32)) and torch.equal(occ, want[1])
    c.synchronize()


def test_many_transparency_queries_in_flight():
    """Twelve streams, each with queries of both kinds on rays of its own, and a
    captured one replayed beside them: every query gives what it gives alone."""
    import torch
    from atlas_rt import ptscene
    c = atlas_rt.Context(device=0)
    try:
        sc = ptscene.build(seed=3, grid=48, n_boxes=20)
        sc["opacity"] = np.linspace(0.0, 0.9, sc["bvh"].n_input).astype(np.float32)
        ptscene.upload(c, sc)
        rng = np.random.default_rng(4)
        jobs = []
        for k in range(12):
            n = int(rng.integers(1, 150_000))
            o = rng.uniform((0, 20, 0), (100, 60, 100), (n, 3)).astype(np.float32)
            d = rng.normal(size=(n, 3)).astype(np.float32)
            rays = torch.from_numpy(scenes.pack_rays(o, d / np.linalg.norm(d, axis=1, keepdims=True))).cuda()
            jobs.append((rays, torch.zeros((n, 8), device="cuda"), torch.zeros(n, device="cuda"), torch.cuda.Stream()))

        def trace(rays, hits, vis, stream):
            c.trace_scene_closest_transparency(rays, 1e-4, 1e4, out=hits, stream=stream.cuda_stream)
            c.trace_scene_any_transparency(rays, 1e-4, 1e4, out=vis, stream=stream.cuda_stream)

        want = []
        for job in jobs:
            trace(*job)
            torch.cuda.synchronize()
            want.append((job[1].clone(), job[2].clone()))
        assert 0.0 < float(torch.cat([v for _, v in want]).mean()) < 1.0
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=jobs[0][3]):
            trace(*jobs[0])
        for _ in range(10):
            for _, hits, vis, _ in jobs:
                hits.zero_()
                vis.zero_()
            torch.cuda.synchronize()
            with torch.cuda.stream(jobs[0][3]):
                graph.replay()
            for job in jobs[1:]:
                trace(*job)
            torch.cuda.synchronize()
            for (_, hits, vis, _), (h, v) in zip(jobs, want):
                assert torch.equal(hits.view(torch.int32), h.view(torch.int32))
                assert torch.equal(vis.view(torch.int32), v.view(torch.int32))
        c.synchronize()
    finally:
        c.close()


@pytest.fixture(scope="module")
def see_through():
    """A scene of partly transparent triangles, 400,100 rays, and their records from
    four launches."""
    import torch
    c = atlas_rt.Context(device=0)
    b = BVH(scenes.random_triangles(3000, seed=13))
    see = b.pack_shading(opacity=np.linspace(-0.2, 0.8, b.n_input).clip(0.0).astype(np.float32))
    mid = c.upload_mesh(b.nodes, b.pack_triangles(), see)
    lo, hi = atlas_rt.mesh_bounds(b)
    c.scene_build(np.array([atlas_rt.make_instance(np.eye(4), mid, atlas_rt.MASK_ALL)]),
                  np.concatenate([lo, hi])[None, :].astype(np.float32))
    total = 400_100
    rays = torch.from_numpy(scenes.pack_rays(*scenes.sphere_rays(total, seed=14))).cuda()
    hits, vis = torch.zeros((total, 8), device="cuda"), torch.zeros(total, device="cuda")
    for at in range(0, total, 100_025):
        c.trace_scene_closest_transparency(rays[at:], 1e-4, 10.0, out=hits[at:], n_rays=100_025)
        c.trace_scene_any_transparency(rays[at:], 1e-4, 10.0, out=vis[at:], n_rays=100_025)
    c.synchronize()
    assert 0.0 < float(vis.mean()) < 1.0
    yield c, rays, hits, vis
    c.close()


@pytest.mark.parametrize("n", [1, 31, 33, 1215, 1216, 1217, 38911, 38913, 136_191, 136_193, 400_009])
def test_transparency_queries_of_any_number_of_rays(see_through, n):
    """Each warp takes its own share of the rays: all of them once, at the edges
    of a warp, of the spread launches and of the grid, and none past n."""
    import torch
    c, rays, hits, vis = see_through
    part, some = torch.full_like(hits, 7.0), torch.full_like(vis, 7.0)
    c.trace_scene_closest_transparency(rays, 1e-4, 10.0, out=part, n_rays=n)
    c.trace_scene_any_transparency(rays, 1e-4, 10.0, out=some, n_rays=n)
    c.synchronize()
    assert torch.equal(part[:n].view(torch.int32), hits[:n].view(torch.int32)) and bool((part[n:] == 7.0).all())
    assert torch.equal(some[:n], vis[:n]) and bool((some[n:] == 7.0).all())
