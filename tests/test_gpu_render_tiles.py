"""Smoothing by tiles (several curvature-flow steps per launch over the tiles with
fluid) against the float32 restatement, bit for bit, where tiles, borders and the
wrapping texture reads can go wrong: images smaller than a tile's border, one pixel
more or less than a tile, step counts that are not a multiple of a launch's, and a
second frame whose fluid lies elsewhere."""
import numpy as np
import pytest

from oracle import render_oracle as RO
from pbf_b200 import render

from test_gpu_render import _blob, _cam

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,iters", [(5, 3, 7), (52, 16, 6), (53, 17, 13), (103, 31, 1), (130, 50, 0)])
def test_smoothing_tile_edges(w, h, iters):
    import torch
    cam = _cam(w, h, iters)
    r = render.Renderer(w, h)
    for pos in (_blob(300, 1), _blob(200, 2) + np.float32([0.25, 0.2, -0.1]), _blob(1, 3) + np.float32(40.0)):
        r.frame(cam, positions=torch.from_numpy(pos).cuda(), stride=3)
        want = RO.render(cam, pos, w, h)
        for name in ("depth_raw", "depth", "thickness", "normal", "room"):
            assert np.array_equal(r.read(name).view(np.uint32), want[name].view(np.uint32)), name
        assert np.abs(r.read("color") - want["color"]).max() <= 2e-5
    r.close()


@pytest.mark.parametrize("between", [1000, 600000])
@pytest.mark.parametrize("iters", [0, 6, 13])
def test_sprites_behind_the_eye(iters, between):
    """Particles nearer to the eye than their radius: sprites whose front lies behind
    the eye have depths below 0, all of window depth 1. The smallest key is kept
    whatever the order of arrival (the second group's blocks start after the first's
    are done: what lies between is behind the eye and draws nothing), and smoothing
    turns such depths into 0, also in tiles without any other."""
    import math
    import torch
    w, h = 210, 50
    cam = render.make_camera((0.0, 0.0, 1.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), math.radians(45.0), w, h, 0.3,
                             smooth_iterations=iters)
    first = np.float32([[-0.1, 0.0, 0.8], [-0.11, 0.01, 0.82], [1.2, 0.3, -3.0]])
    second = np.float32([[-0.12, 0.0, 0.78], [-0.1, 0.02, 0.81], [-0.11, 0.0, 0.82], [1.6, -0.3, -4.0]])
    unseen = np.full((between, 3), 2.0, np.float32)
    r = render.Renderer(w, h)
    r.frame(cam, positions=torch.from_numpy(np.concatenate([first, unseen, second])).cuda(), stride=3)
    want = RO.render(cam, np.concatenate([first, second]), w, h)
    tiles = [want["depth_raw"][y:y + 16, x:x + 52] for y in range(0, h, 16) for x in range(0, w, 52)]
    assert any((t < 0).any() and not (t > 0).any() for t in tiles)
    for name in ("depth_raw", "depth", "thickness", "normal", "room"):
        assert np.array_equal(r.read(name).view(np.uint32), want[name].view(np.uint32)), name
    assert np.abs(r.read("color") - want["color"]).max() <= 2e-5
    r.close()


@pytest.mark.parametrize("n", [151551, 151552])
def test_sprites_of_few_and_of_many_particles(n):
    """From 151,552 particles (148 SMs x 1,024) on, the sprite pass reads a pixel before it
    writes it. All but 300 are behind the eye, which draws nothing."""
    import torch
    w, h = 97, 61
    cam = _cam(w, h, 6, radius=0.05)
    seen = _blob(300, 4)
    pos = np.full((n, 3), 50.0, np.float32)
    pos[:: n // 300][:300] = seen
    r = render.Renderer(w, h)
    r.frame(cam, positions=torch.from_numpy(pos).cuda(), stride=3)
    want = RO.render(cam, seen, w, h)
    for name in ("depth_raw", "depth", "thickness", "normal"):
        assert np.array_equal(r.read(name).view(np.uint32), want[name].view(np.uint32)), name
    r.close()
