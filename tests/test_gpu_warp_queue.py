"""The warp-level triangle queue of the persistent traversal at its edges.

Every ray's answer is the minimum of (t, depth-first slot) over its candidates whichever lane of the
warp tests them, so hits must equal the oracle's bit for bit: scenes whose nodes hand a lane up to 24
triangles at once (coincident primitives, every t tied), batches that leave a warp mostly empty, and
a wavefront whose lanes walk different scenes.
"""
import numpy as np
import pytest

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi, scenes

pytestmark = pytest.mark.gpu


def _stack_scene(copies):
    """`copies` coincident copies of a small mesh, and a sphere: leaves of that many primitives."""
    sb = scenes.SceneBuilder()
    m = sb.material(sb.layered_bsdf(sb.lambertian()))
    tris = scenes.displaced_icosphere(1, radius=0.5, seed=3)
    for _ in range(copies):
        sb.triangles(tris, m)
    sb.sphere((0.9, 0.1, 0.0), 0.3, m)
    return sb


@pytest.mark.parametrize("copies", [1, 2, 3, 4, 24, 25, 40])
@pytest.mark.parametrize("n", [1, 31, 33, 2000])
def test_coincident_primitives_and_small_batches(device, oracle, copies, n):
    packed = _stack_scene(copies).build()
    gs = spt.GpuScene(device, packed)
    rays = scenes.incoherent_rays(n, seed=copies, half_extent=1.2)
    got = gs.intersect(rays)["hits"]
    exp = oracle.scene(packed).intersect(rays)["hits"]
    gs.close()
    np.testing.assert_array_equal(got["prim_id"], exp["prim_id"])
    hit = exp["prim_id"] != abi.SPT_MISS
    np.testing.assert_array_equal(got["t"][hit].view(np.uint32), exp["t"][hit].view(np.uint32))


def test_lanes_of_one_warp_on_different_scenes(device):
    """A batch whose jobs are of several scenes, of so few paths each that a warp holds rays of all
    of them, equals the single renders (a render's image does not depend on the batch it is in, up
    to the order of its float additions: at most 5 bounces times 4 samples of relative 2^-24 each)."""
    import torch
    cams = [scenes.box_camera(9, 7), scenes.furnace_camera(8, 8), scenes.displaced_mesh_camera(11, 5)]
    built = [scenes.box_scene(3), scenes.furnace_scene("coating"), _stack_scene(5)]
    jobs, single = [], []
    for i, (sb, cam) in enumerate(zip(built, cams)):
        gs = spt.GpuScene(device, sb.build())
        p = scenes.pt_params(spp=4, sampler="jittered", termination="max-length", path_length=5, seed=40 + i)
        jobs.append((gs, cam, p))
        single.append(gs.pathtrace(cam, p)[0])
    bufs = [torch.zeros((c.height, c.width, 3), dtype=torch.float32, device="cuda") for c in cams]
    spt.render_batch(device, jobs, [b.data_ptr() for b in bufs])
    for b, s in zip(bufs, single):
        np.testing.assert_allclose(b.cpu().numpy(), s, rtol=2e-6, atol=1e-7)
