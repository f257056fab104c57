"""Scenes of very many materials: materials that share a layered BSDF share its layers on the device, and more
materials than a primitive's 30-bit number can name are numbered anew."""
import ctypes as C

import numpy as np
import pytest

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi, scenes

pytestmark = pytest.mark.gpu

CAM = dict(kind="pinhole", position=(0.0, 0.2, 3.0), look_at=(0, 0, 0), fov=50.0, width=48, height=40)
PARAMS = dict(spp=4, sampler="jittered", termination="max-length", path_length=4, seed=5)


def _builder(n_extra, layers=2):
    """A ball and a sphere of two materials on one stack, with n_extra unused materials between them."""
    sb = scenes.SceneBuilder(background=(0.5, 0.6, 0.7))
    top = sb.smooth_dielectric(ior=1.5)
    stack = sb.layered_bsdf(*([top] * (layers - 1) + [sb.lambertian(kd=(0.7, 0.4, 0.2))]))
    plain = sb.layered_bsdf(sb.cook_torrance(roughness=0.3))
    a = sb.material(stack, emission=(0.1, 0.0, 0.0))
    sb.materials += [(stack, (0.0, 0.0, 0.0))] * n_extra
    b = sb.material(stack, emission=(0.0, 0.2, 0.0))
    c = sb.material(plain, emission=(0.0, 0.0, 0.3))
    sb.triangles(scenes.displaced_icosphere(2, radius=0.6), a)
    sb.sphere((0.8, 0.1, 0.3), 0.35, b)
    sb.sphere((-0.8, 0.0, 0.2), 0.3, c)
    return sb


def _image(device, packed):
    gs = spt.GpuScene(device, packed)
    img, _ = gs.pathtrace(scenes.camera(**CAM), scenes.pt_params(**PARAMS))
    size = gs.device_bytes()
    gs.close()
    return img, size


def test_materials_share_their_layers(device):
    few, small = _image(device, _builder(0, layers=40).build())
    many, large = _image(device, _builder(50000, layers=40).build())
    # the same 4 samples a pixel, added in any order
    np.testing.assert_allclose(many, few, rtol=4 * 2.0 ** -23, atol=1e-7)
    assert large - small < 50000 * 64   # a material's own record, no layers


def test_more_materials_than_thirty_bits(device):
    """2^30 + 2 materials: the table of zeros between the first and the last two is never touched."""
    ref, _ = _image(device, _builder(0).build())
    sb = _builder(0)
    packed = sb.build()
    n = (1 << 30) + 2
    dt = np.dtype([("layered", np.uint32), ("emission", np.float32, 3)])
    assert dt.itemsize == C.sizeof(abi.Material)
    table = np.zeros(n, dt)
    mats = np.frombuffer(packed.materials, dt, 3)
    table[0], table[n - 2], table[n - 1] = mats[0], mats[1], mats[2]
    packed.mats[:] = np.where(packed.mats == 0, 0, packed.mats + (n - 3)).astype(np.uint32)
    packed.desc.materials = C.cast(table.ctypes.data, C.POINTER(abi.Material))
    packed.desc.n_materials = n
    img, _ = _image(device, packed)
    np.testing.assert_allclose(img, ref, rtol=4 * 2.0 ** -23, atol=1e-7)
