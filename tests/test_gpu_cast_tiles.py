"""The tiled ray-caster kernel at the edges of its 16 x 8 pixel blocks and 8 x 4 pixel warps.

A warp's lanes outside the image hold no ray and help with the others' triangles; its last four rays get
eight lanes each.  Images must equal the oracle's bit for bit, as every caster's do.
"""
import numpy as np
import pytest

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def smooth(device, oracle):
    packed = scenes.smooth_mesh_scene(3).build()     # flat and smooth triangles and a sphere
    gs = spt.GpuScene(device, packed)
    yield gs, oracle.scene(packed)
    gs.close()


@pytest.mark.parametrize("size", [(1, 1), (8, 4), (9, 5), (16, 8), (17, 9), (3, 33), (129, 2)])
@pytest.mark.parametrize("mode", [abi.RAYCAST_NORMAL, abi.RAYCAST_DEPTH, abi.RAYCAST_COUNT])
def test_ragged_images(smooth, size, mode):
    gs, osc = smooth
    cam = scenes.box_camera(*size)
    got = gs.raycast(cam, mode)
    exp, _ = osc.raycast(cam, mode)
    assert got.tobytes() == np.ascontiguousarray(exp).tobytes()
