"""Training steps with no records at all, and with fewer records than steps:
the gradients are cleared behind a kernel that has nothing to add to them."""
import numpy as np
import pytest

import atlas_rt
from atlas_rt import ptscene, scenes
from test_rc_gpu import HI, LO, random_records

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    c = atlas_rt.Context(device=0)
    ptscene.upload(c, ptscene.build(seed=7, grid=16, n_boxes=4))
    yield c
    c.close()


@pytest.mark.parametrize("log2_table", [10, 14, 19])
@pytest.mark.parametrize("steps", [1, 4])
def test_frames_whose_paths_hit_nothing_leave_the_parameters(scene, log2_table, steps):
    """Gradients into host memory leave the cache's own buffers full; a frame
    that looks at the sky then trains on nothing: the loss is 0, and Adam,
    whose moments are still 0, changes no parameter."""
    import torch
    rc = atlas_rt.RadianceCache(scene, LO, HI, log2_table=log2_table, seed=5)
    try:
        sky = atlas_rt.make_camera(scenes.pinhole_camera(64, 48, eye=(50.0, 200.0, 50.0), target=(60.0, 400.0, 50.0)))
        q = torch.from_numpy(random_records(3000, 6)).cuda()
        before = rc.get_params()
        for frame in range(3):
            gm, gg = np.zeros(rc.n_mlp, np.float32), np.zeros(rc.n_grid, np.float32)
            rc.gradients(q, gm, gg)
            assert gm.any() and gg.any()
            assert rc.train_frame(sky, frame, n_paths=512, steps=steps, want_loss=True) == 0.0
            for a, b in zip(before, rc.get_params()):
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    finally:
        rc.close()


def test_frames_of_fewer_records_than_steps(scene):
    """Eight paths in eight steps, half of them past the scene's edge: every
    step's slice holds a few records or none."""
    rc = atlas_rt.RadianceCache(scene, LO, HI, log2_table=14, seed=5)
    try:
        edge = atlas_rt.make_camera(scenes.pinhole_camera(64, 48, eye=(50.0, 200.0, 50.0), target=(300.0, 150.0, 50.0)))
        losses = [rc.train_frame(edge, f, n_paths=8, steps=8, max_bounces=1, want_loss=True) for f in range(30)]
        assert np.isfinite(losses).all() and min(losses) == 0.0
        assert all(np.isfinite(a).all() for a in rc.get_params())
    finally:
        rc.close()
