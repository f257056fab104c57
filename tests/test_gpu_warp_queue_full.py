"""The warp-level triangle queue with full warps: at least 32 rays a warp, so that the warps walk and queue
(smaller batches are spread one ray a warp and end in the eight-lanes-a-ray loop at once).  Steps that find
more triangles than the queue has room for, warps whose lanes walk different scenes, and renders in two
waves over several scenes."""
import numpy as np
import pytest
import torch

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi, scenes
from test_gpu_warp_queue import _stack_scene

pytestmark = pytest.mark.gpu


def _aimed_rays(n, seed):
    """Rays from around the stack of coincident meshes into it: nearly every one meets leaves of all copies."""
    g = np.random.default_rng(seed)
    o = g.standard_normal((n, 3))
    o *= 1.5 / np.linalg.norm(o, axis=1, keepdims=True)
    d = 0.4 * g.uniform(-1.0, 1.0, (n, 3)) - o
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = o
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    return r


@pytest.mark.parametrize("copies,n", [(1, 300007), (8, 300007), (24, 1 << 18), (25, (1 << 18) + 1), (40, 300007)])
def test_steps_that_overfill_the_queue(device, oracle, copies, n):
    packed = _stack_scene(copies).build()
    gs = spt.GpuScene(device, packed)
    rays = _aimed_rays(n, copies)
    d_rays = torch.from_numpy(rays).cuda()
    hits, again = (torch.empty((n, 4), dtype=torch.int32, device="cuda") for _ in range(2))
    gs.intersect_device(d_rays.data_ptr(), n, hits.data_ptr(), 0)
    # backwards: other rays side by side in a warp
    d_back = d_rays.flip(0).contiguous()
    gs.intersect_device(d_back.data_ptr(), n, again.data_ptr(), 0)
    torch.cuda.synchronize()
    gs.close()
    exp = oracle.scene(packed).intersect(rays)["hits"]
    hit = exp["prim_id"] != abi.SPT_MISS
    assert hit.mean() > 0.9
    for got in (hits.cpu().numpy(), again.flip(0).cpu().numpy()):
        np.testing.assert_array_equal(got[:, 1].view(np.uint32), exp["prim_id"])
        np.testing.assert_array_equal(got[hit, 0], exp["t"][hit].view(np.int32))


def _kinds():
    return [(scenes.box_scene(3), scenes.box_camera(5, 4)), (scenes.furnace_scene("coating"), scenes.furnace_camera(5, 4)),
            (_stack_scene(5), scenes.displaced_mesh_camera(5, 4))]


# A pixel is 4 samples of at most 5 positive contributions, added up in any order.
SUM_TOL = dict(rtol=20 * 2.0 ** -24, atol=1e-7)


@pytest.mark.parametrize("sort", [0, 1, 2])
def test_a_warp_of_many_scenes(device, sort):
    """1,800 jobs of 80 paths, scene by scene in turn: 144,000 paths, so that every warp of the chip takes 32
    at a time and a chunk spans two jobs."""
    p = scenes.pt_params(spp=4, sampler="jittered", termination="max-length", path_length=5, seed=44)
    built = [(spt.GpuScene(device, sb.build()), cam) for sb, cam in _kinds()]
    single = [gs.pathtrace(cam, p)[0] for gs, cam in built]
    n = 1800
    jobs = [(*built[i % 3], p) for i in range(n)]
    out = torch.zeros((n, 4, 5, 3), dtype=torch.float32, device="cuda")
    tune = spt.default_tune()
    tune.sort_shading = sort
    spt.render_batch(device, jobs, [out[i].data_ptr() for i in range(n)], tune=tune)
    got = out.cpu().numpy()
    for i in range(n):
        np.testing.assert_allclose(got[i], single[i % 3], **SUM_TOL)
    for gs, _ in built:
        gs.close()


@pytest.mark.parametrize("capacity", [1024, 4099, 20001])
@pytest.mark.parametrize("end", ["max-length", "russian-roulette"])
def test_two_waves_over_several_scenes(device, capacity, end):
    """More paths than the pool, an odd number of both: two waves, split inside a job, on the persistent
    traversal.  Each image is the single render's."""
    cams = [scenes.box_camera(37, 29), scenes.furnace_camera(41, 41), scenes.displaced_mesh_camera(53, 31)]
    jobs, single = [], []
    for i, ((sb, _), cam) in enumerate(zip(_kinds(), cams)):
        gs = spt.GpuScene(device, sb.build())
        p = scenes.pt_params(spp=9 if i else 1, sampler="jittered", termination=end, path_length=3, seed=60 + i)
        jobs.append((gs, cam, p))
        single.append(gs.pathtrace(cam, p))
    total = sum(int(st.paths) for _, st in single)
    assert total % 2 == 1 and total > capacity
    tune = spt.default_tune()
    tune.capacity, tune.traversal = capacity, 2
    bufs = [torch.zeros((c.height, c.width, 3), dtype=torch.float32, device="cuda") for c in cams]
    st = spt.render_batch(device, jobs, [b.data_ptr() for b in bufs], tune=tune)
    assert st[0].segments == sum(int(s.segments) for _, s in single)
    for b, (img, _) in zip(bufs, single):
        # under roulette a path may go on: its terms still add up along one thread, the pixel's 9 samples do not
        np.testing.assert_allclose(b.cpu().numpy(), img, rtol=45 * 2.0 ** -24, atol=1e-7)
    for gs, _, _ in jobs:
        gs.close()
