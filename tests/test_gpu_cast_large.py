"""Normal and depth images on both sides of 6 pixels a triangle, where the casters of larger scenes go over from
the tiled kernel to one thread per pixel, against the reference's traversal (the image with
statistics)."""
import pytest

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh(device):
    packed = scenes.displaced_mesh_scene(7).build()
    assert packed.n_prims == 327680   # 1,966,080 pixels
    gs = spt.GpuScene(device, packed)
    yield gs
    gs.close()


@pytest.mark.parametrize("size", [(1092, 1800), (1093, 1800), (1024, 1920), (1025, 1919), (1023, 1921), (1025, 1921)])
@pytest.mark.parametrize("mode", [abi.RAYCAST_NORMAL, abi.RAYCAST_DEPTH])
def test_route(mesh, size, mode):
    cam = scenes.camera("pinhole", position=(0.35, 0.4, 3.0), look_at=(0, 0, 0), fov=40.0, width=size[0], height=size[1])
    got = mesh.raycast(cam, mode)
    exp, _ = mesh.raycast(cam, mode, stats=True)
    assert got.tobytes() == exp.tobytes()
