"""ae_rt_mesh_get_bvh into host and device memory: the library keeps its nodes
in an order of its own and hands them out in the engine's, 524,288 at a time
where a copy is needed."""
import numpy as np
import pytest

import atlas_rt
from atlas_rt import BVH, _native, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 1000, 524_288, 524_289, 524_290, 1_200_001])
def test_built_nodes_into_host_and_device_memory(ctx, n):
    import torch
    mid, _ = ctx.build_mesh(scenes.random_triangles(n, seed=3))
    nodes, _ = ctx.mesh_bvh(mid)
    assert len(nodes) == n - 1
    words = nodes.view(np.int32).reshape(-1, 16)
    dev = torch.zeros(16 * (n + 1), dtype=torch.int32, device="cuda")
    for first in (0, 16, 3):            # words: aligned to 16 bytes, and to 4 alone
        dev.fill_(7)
        assert _native.lib().ae_rt_mesh_get_bvh(ctx.handle, mid, dev[first:].data_ptr(), None, None, None) == 0
        torch.cuda.synchronize()
        got, end = dev.cpu().numpy(), first + 16 * (n - 1)
        assert np.array_equal(got[first:end].reshape(-1, 16), words)
        assert (got[:first] == 7).all() and (got[end:] == 7).all()
    # a tree over every triangle: each child box lies in its parent's
    child = words[:, 12:14]
    box = words.view(np.float32)[:, :12].reshape(-1, 2, 6)
    assert ((child >= -n) & (child < n - 1)).all()
    for side in (0, 1):
        inner = child[:, side] >= 0
        below = box[child[inner, side]]
        assert (below[..., :3] >= box[inner, side, None, :3]).all() and (below[..., 3:] <= box[inner, side, None, 3:]).all()


def test_uploaded_nodes_come_back(ctx):
    b = BVH(scenes.random_triangles(70_000, seed=4))
    gt = b.pack_triangles()
    nodes, tris = ctx.mesh_bvh(ctx.upload_mesh(b.nodes, gt))
    got, want = (np.ascontiguousarray(a).view(np.uint32).reshape(-1, 16) for a in (nodes, b.nodes))
    assert np.array_equal(got[:, :14], want[:, :14]) and np.array_equal(tris, gt)
