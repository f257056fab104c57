"""Rays whose origins lie thousands of units from a fine mesh: the rounding of a box plane's distance is then
as large as the 1e-3 by which the reference's boxes are inflated.  The 8-wide box tests allow for their own
rounding, so no hit that the reference's traversal finds is lost.  (From there on the reference's own box
test loses hits, so a nearer one than its is no error.)"""
import numpy as np
import pytest
import torch

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi, scenes

pytestmark = pytest.mark.gpu

N = 1 << 22


@pytest.fixture(scope="module")
def mesh(device):
    gs = spt.GpuScene(device, scenes.displaced_mesh_scene(8).build())
    yield gs
    gs.close()


def _unit(g):
    v = torch.randn((N, 3), generator=g, device="cuda", dtype=torch.float64)
    return v / v.norm(dim=1, keepdim=True)


@pytest.mark.parametrize("distance", [3, 300, 3000, 6000, 8000])
def test_no_hit_is_lost(mesh, distance):
    g = torch.Generator(device="cuda").manual_seed(distance)
    rays = torch.zeros((N, 8), device="cuda")
    rays[:, 0:3] = (_unit(g) * distance).float()
    target = _unit(g) * torch.rand((N, 1), generator=g, device="cuda", dtype=torch.float64)
    d = target - rays[:, 0:3].double()
    rays[:, 4:7] = (d / d.norm(dim=1, keepdim=True)).float()
    hits, ref = (torch.empty((N, 4), dtype=torch.int32, device="cuda") for _ in range(2))
    tests = torch.empty(N, dtype=torch.int32, device="cuda")
    mesh.intersect_device(rays.data_ptr(), N, hits.data_ptr(), 0)
    mesh.count_device(rays.data_ptr(), N, ref.data_ptr(), tests.data_ptr(), None)   # the reference's traversal
    torch.cuda.synchronize()
    t, t_ref = hits[:, 0].view(torch.float32), ref[:, 0].view(torch.float32)
    assert int((t > t_ref).sum()) == 0
    assert int((ref[:, 1] != -1).sum()) > 0.9 * N and abi.SPT_MISS == 0xFFFFFFFF
    if distance <= 300:
        assert torch.equal(hits[:, 0:2], ref[:, 0:2])


@pytest.mark.parametrize("distance", [3, 300, 3000, 6000])
def test_small_batches_too(mesh, distance):
    """A few rays per warp, eight lanes each; and the ray casters' one thread per pixel and tiles."""
    w = 1920
    cam = scenes.camera("pinhole", position=(0.2 * distance, 0.3 * distance, 0.93 * distance), look_at=(0, 0, 0),
                        fov=float(np.degrees(2.0 * np.arctan(0.9 / distance))), width=w, height=w)
    depth = mesh.raycast(cam, abi.RAYCAST_DEPTH)
    ref, _ = mesh.raycast(cam, abi.RAYCAST_DEPTH, stats=True)   # the reference's traversal
    far = np.inf
    assert np.count_nonzero(np.where(depth < 0, far, depth) > np.where(ref < 0, far, ref)) == 0
    g = torch.Generator(device="cuda").manual_seed(distance + 1)
    o = np.array([0.2, 0.3, 0.93]) * distance
    for n in (1000, 20011):
        target = (_unit(g)[:n] * 0.9).cpu().numpy()
        rays = np.zeros((n, 8), np.float32)
        rays[:, 0:3] = o
        d = target - rays[:, 0:3].astype(np.float64)
        rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
        dev = torch.from_numpy(rays).cuda()
        hits, ref_h = (torch.empty((n, 4), dtype=torch.int32, device="cuda") for _ in range(2))
        mesh.intersect_device(dev.data_ptr(), n, hits.data_ptr(), 0)
        mesh.count_device(dev.data_ptr(), n, ref_h.data_ptr(), None, None)
        torch.cuda.synchronize()
        assert int((hits[:, 0].view(torch.float32) > ref_h[:, 0].view(torch.float32)).sum()) == 0
