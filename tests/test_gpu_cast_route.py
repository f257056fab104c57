"""Ray-caster images on both sides of the choice between the tiled kernel and one thread per pixel: by the
scene's size (more than 2,048 primitives) and, below 131,072, by the image's (500,000 pixels)."""
import numpy as np
import pytest

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("subdiv,size", [(2, (17, 9)), (4, (17, 9)), (4, (129, 2)), (4, (801, 625)), (4, (800, 624))])
@pytest.mark.parametrize("mode", [abi.RAYCAST_NORMAL, abi.RAYCAST_DEPTH])
def test_route(device, oracle, subdiv, size, mode):
    packed = scenes.smooth_mesh_scene(subdiv).build()
    gs = spt.GpuScene(device, packed)
    cam = scenes.box_camera(*size)
    got = gs.raycast(cam, mode)
    exp, _ = oracle.scene(packed).raycast(cam, mode)
    assert got.tobytes() == np.ascontiguousarray(exp).tobytes()
    gs.close()
