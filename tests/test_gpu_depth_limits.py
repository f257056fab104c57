"""Renders within one pool under a depth limit: iterations are launched for paths that live, not for the
limit.  Every limit gives the image of the host-driven loop."""
import time

import numpy as np
import pytest
import torch

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi, native, scenes

pytestmark = pytest.mark.gpu


def _image(device, gs, cam, p, tune=None):
    buf = torch.zeros((cam.height, cam.width, 3), dtype=torch.float32, device="cuda")
    st = spt.render_batch(device, [(gs, cam, p)], [buf.data_ptr()], tune=tune)
    return buf.cpu().numpy(), st[0].segments


def test_time_follows_the_paths_not_the_limit(device):
    """Every path ends at its second vertex: a limit of 64 costs no more than one of 16."""
    gs = spt.GpuScene(device, scenes.furnace_scene("lambertian").build())
    cam = scenes.furnace_camera(64, 64)
    img = torch.zeros((64, 64, 3), dtype=torch.float32, device="cuda")
    best = {}
    for limit in (16, 64):
        p = scenes.pt_params(spp=4, termination="max-length", path_length=limit, seed=3)
        times = []
        for _ in range(30):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            gs.pathtrace_device(cam, p, img.data_ptr())
            times.append(time.perf_counter() - t0)
        best[limit] = min(times)
    gs.close()
    # 64 launched iterations take three times as long as 16; a look at the counters a twentieth
    assert best[64] <= 1.5 * best[16], best


@pytest.mark.parametrize("limit", [1, 2, 8, 9, 15, 16, 17, 18, 33, 64, 65])
def test_every_limit_gives_the_same_image(device, limit):
    """Against the host-driven loop, up to the order of the pixels' float additions: 4 samples, each a sum
    along its path, of positive terms."""
    gs = spt.GpuScene(device, scenes.box_scene(3).build())
    cam = scenes.box_camera(40, 33)
    p = scenes.pt_params(spp=4, sampler="jittered", termination="max-length", path_length=limit, seed=limit)
    t = spt.default_tune()
    t.host_loop = 1
    (got, n), (exp, m) = _image(device, gs, cam, p), _image(device, gs, cam, p, t)
    gs.close()
    assert n == m
    np.testing.assert_allclose(got, exp, rtol=4 * 2.0 ** -23, atol=1e-7)


@pytest.mark.parametrize("budget,limit", [(1, 40), (8, 40), (9, 40), (16, 40)])
def test_the_budget_still_ends_the_render(device, budget, limit):
    gs = spt.GpuScene(device, scenes.box_scene(3).build())
    t = spt.default_tune()
    t.max_iterations = budget
    with pytest.raises(native.SptError) as e:
        _image(device, gs, scenes.box_camera(64, 48), scenes.pt_params(spp=16, path_length=limit, seed=9), t)
    assert e.value.status == abi.SPT_ERR_TIMEOUT
    gs.close()
