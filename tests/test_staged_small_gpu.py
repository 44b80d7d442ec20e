"""Staged launches (tiles of 16 rays through shared memory) of fewer rays than
fill the GPU: every lane takes rays of its warp's tile, and the records are
the plain loads'."""
import numpy as np
import pytest

import atlas_rt
from atlas_rt import BVH, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def contexts():
    b = BVH(scenes.random_triangles(20000, seed=51))
    gt, (lo, hi) = b.pack_triangles(), atlas_rt.mesh_bounds(b)
    made = []
    for staged in (False, True):
        c = atlas_rt.Context(device=0, staged_rays=staged)
        mid = c.upload_mesh(b.nodes, gt)
        c.scene_build(np.array([atlas_rt.make_instance(np.eye(4), mid, atlas_rt.MASK_ALL)]),
                      np.concatenate([lo, hi])[None, :].astype(np.float32))
        made.append((c, mid))
    yield made, scenes.pack_rays(*scenes.sphere_rays(40000, seed=52))
    for c, _ in made:
        c.close()


@pytest.mark.parametrize("n", [100, 1215, 1216, 1217, 5000, 19456, 38913])
def test_small_staged_launches_equal_plain_loads(contexts, n):
    made, rays = contexts
    out = [(c.trace_closest(m, rays, 1e-4, 10.0, n_rays=n), c.trace_any(m, rays, 1e-4, 10.0, n_rays=n),
            c.trace_scene_closest(rays, 1e-4, 10.0, n_rays=n), c.trace_scene_any(rays, 1e-4, 10.0, n_rays=n))
           for c, m in made]
    for plain, staged in zip(*out):
        assert np.array_equal(plain[:n].view(np.uint8), staged[:n].view(np.uint8))
    assert out[0][1][:n].any()
