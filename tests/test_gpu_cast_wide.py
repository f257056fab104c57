"""The tiled normal and depth casters (scenes of more than 2,048 primitives): at the edges of their 16 x 8
pixel blocks and 8 x 4 pixel warps against the oracle, and the full-HD images of the 1.31M-triangle mesh
without statistics, which take other kernels than those with, against the reference's own images."""
import hashlib

import numpy as np
import pytest

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi, scenes
from test_gpu_config_pins import CONFIGS

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def smooth(device, oracle):
    packed = scenes.smooth_mesh_scene(4).build()     # flat and smooth triangles and a sphere
    assert packed.n_prims > 2048
    gs = spt.GpuScene(device, packed)
    yield gs, oracle.scene(packed)
    gs.close()


@pytest.mark.parametrize("size", [(1, 1), (2, 1), (4, 1), (5, 1), (8, 4), (9, 5), (16, 8), (17, 9), (3, 33), (129, 2), (63, 65)])
@pytest.mark.parametrize("mode", [abi.RAYCAST_NORMAL, abi.RAYCAST_DEPTH])
@pytest.mark.parametrize("view", ["box", "outside", "orthographic"])
def test_ragged_images(smooth, size, mode, view):
    gs, osc = smooth
    w, h = size
    if view == "box":
        cam = scenes.box_camera(w, h)
    elif view == "outside":   # most rays miss the root box
        cam = scenes.camera("pinhole", position=(0.5, 0.5, 2.35), look_at=(0.9, 0.9, 0.0), fov=70.0, width=w, height=h)
    else:                     # axis-parallel rays
        cam = scenes.camera("orthographic", position=(0.5, 0.5, 6), look_at=(0.5, 0.5, 0), width=w, height=h,
                            window=(-0.5, 0.5, -0.5, 0.5))
    got = gs.raycast(cam, mode)
    exp, _ = osc.raycast(cam, mode)
    assert got.tobytes() == np.ascontiguousarray(exp).tobytes()


@pytest.fixture(scope="module")
def mesh(device):
    gs = spt.GpuScene(device, scenes.displaced_mesh_scene(8).build())
    yield gs
    gs.close()


@pytest.mark.parametrize("name,mode", [("normal", abi.RAYCAST_NORMAL), ("depth", abi.RAYCAST_DEPTH),
                                       ("count", abi.RAYCAST_COUNT)])
def test_full_hd_images_without_statistics(mesh, name, mode):
    img = mesh.raycast(scenes.displaced_mesh_camera(1920, 1080), mode)
    assert hashlib.sha256(np.ascontiguousarray(img).tobytes()).hexdigest() == CONFIGS["c1"]["images"][name]["sha256"]
