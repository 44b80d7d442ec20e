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
