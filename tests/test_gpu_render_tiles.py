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
