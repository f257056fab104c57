"""Renders larger than the pool on both sides of the choice between one wave and two: two for at least two
pools of paths where a scene has layered stacks, for at least 32 where none has, always on a traversal of one
thread per path.  The image is that of a pool
that holds every path, up to the order of a pixel's float additions."""
import numpy as np
import pytest
import torch

import swpathtracer_b200 as spt
from swpathtracer_b200 import scenes

pytestmark = pytest.mark.gpu

POOL = 1024


@pytest.mark.parametrize("layered", [False, True])
@pytest.mark.parametrize("size,spp", [((64, 16), 1), ((41, 25), 1), ((64, 32), 1), ((64, 31), 1), ((43, 27), 9),
                                      ((64, 57), 9), ((61, 60), 9)])
@pytest.mark.parametrize("end,traversal", [("max-length", 2), ("russian-roulette", 2), ("max-length", 1),
                                           ("russian-roulette", 0)])
def test_images_do_not_depend_on_the_waves(device, layered, size, spp, end, traversal):
    sb = scenes.furnace_scene("coating") if layered else scenes.box_scene(3)
    cam = scenes.furnace_camera(*size) if layered else scenes.box_camera(*size)
    gs = spt.GpuScene(device, sb.build())
    p = scenes.pt_params(spp=spp, sampler="jittered", termination=end, path_length=4, max_depth=12, seed=7)
    out = []
    for capacity in (1 << 20, POOL):
        tune = spt.default_tune()
        tune.capacity, tune.traversal = capacity, traversal
        img = torch.zeros((cam.height, cam.width, 3), dtype=torch.float32, device="cuda")
        st = spt.render_batch(device, [(gs, cam, p)], [img.data_ptr()], tune=tune)
        out.append((img.cpu().numpy(), st[0].segments))
    gs.close()
    assert out[0][1] == out[1][1]
    # 9 samples of at most 12 positive terms, each a sum along its path
    np.testing.assert_allclose(out[1][0], out[0][0], rtol=(9 + 12) * 2.0 ** -23, atol=1e-7)
