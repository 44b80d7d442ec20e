"""Path-traced images and tiles of fewer pixels than a block has threads: the
bits of the same pixels in a larger image, whatever the calls before left in
the context's counters and queues."""
import numpy as np
import pytest

import atlas_rt
from atlas_rt import ptscene, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tracer():
    c = atlas_rt.Context(device=0)
    ptscene.upload(c, ptscene.build(seed=7, grid=16, n_boxes=4))
    yield c
    c.close()


@pytest.mark.parametrize("bounces", [3, 64, 300])
@pytest.mark.parametrize("w,h", [(1, 1), (1, 7), (5, 3), (8, 8), (15, 17)])
def test_tiles_of_few_pixels(tracer, w, h, bounces):
    """A tile that sets 4 (bounces + 2) counters from fewer pixels than that,
    after the whole image of 408 pixels has left its own counts in them."""
    import torch
    cam = atlas_rt.make_camera(scenes.pinhole_camera(24, 17))
    whole, tile = (torch.zeros((24 * 17, 4), device="cuda") for _ in range(2))
    tracer.pathtrace(cam, whole, spp=2, max_bounces=bounces)
    x, y = (24 - w) // 2, (17 - h) // 2
    for _ in range(2):              # the second call finds what the first left
        tile.zero_()
        tracer.pathtrace(cam, tile, spp=2, max_bounces=bounces, tile=(x, y, w, h))
    tracer.synchronize()
    whole, tile = (a.cpu().numpy().reshape(17, 24, 4) for a in (whole, tile))
    assert np.array_equal(tile[y:y + h, x:x + w], whole[y:y + h, x:x + w]) and whole[..., :3].max() > 0
    tile[y:y + h, x:x + w] = 0
    assert not tile.any()


@pytest.mark.parametrize("bounces", [3, 64])
@pytest.mark.parametrize("w,h", [(1, 1), (1, 7), (5, 3)])
def test_images_of_few_pixels(tracer, w, h, bounces):
    """The first h rows of an image 2^k times as high through the same pixels
    (its vertical span 2^k times as long, so every ray has the same bits)."""
    import torch
    f = 1
    while w * h * f < 512:
        f *= 2
    small = {**scenes.pinhole_camera(w, h), "jitter": (0.0, 0.0)}
    tall = {**small, "height": h * f, "bottom": np.asarray(small["bottom"], np.float32) * np.float32(f)}
    out = {}
    for name, cam in (("tall", tall), ("small", small), ("again", small)):
        n = cam["width"] * cam["height"]
        acc = torch.zeros((n, 4), device="cuda")
        frame = torch.zeros((3, n), dtype=torch.int32, device="cuda")
        tracer.pathtrace(atlas_rt.make_camera(cam), acc, spp=2, max_bounces=bounces)
        tracer.pathtrace_realtime(atlas_rt.make_camera(cam), frame, max_radiance=10.0, spp=2, max_bounces=bounces)
        tracer.synchronize()
        out[name] = acc.cpu().numpy(), frame.cpu().numpy()
    for name in ("small", "again"):
        assert np.array_equal(out[name][0], out["tall"][0][:w * h])
        assert np.array_equal(out[name][1], out["tall"][1][:, :w * h])
    assert out["small"][0].any()       # (the one centred pixel of the 1 x 1 real-time image is black)
