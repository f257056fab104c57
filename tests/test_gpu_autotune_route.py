"""The autotuner names the traversal it timed: a render takes none that a scene of its batch does not have."""
import pytest

import swpathtracer_b200 as spt
from swpathtracer_b200 import scenes

pytestmark = pytest.mark.gpu


def _job(device, sb):
    return spt.GpuScene(device, sb.build()), scenes.box_camera(32, 24), scenes.pt_params(spp=4, path_length=3, seed=2)


def _without_a_tree():
    sb = scenes.SceneBuilder(acceleration_structure="none")
    m = sb.material(sb.layered_bsdf(sb.lambertian()), emission=(0.2, 0.2, 0.2))
    sb.triangles(scenes.displaced_icosphere(1, radius=0.4, center=(0.5, 0.5, 0.5)), m)
    return sb


@pytest.mark.parametrize("env,builders,highest", [
    (None, [_without_a_tree], 0),
    (None, [lambda: scenes.box_scene(2), _without_a_tree], 0),
    ("binary", [lambda: scenes.box_scene(2)], 0),
    ("wide", [lambda: scenes.box_scene(2)], 1),
    (None, [lambda: scenes.box_scene(2)], 2),
])
def test_the_result_names_a_traversal_the_batch_has(device, monkeypatch, env, builders, highest):
    if env:
        monkeypatch.setenv("SPT_TRAVERSAL", env)
    jobs = [_job(device, b()) for b in builders]
    got = [spt.autotune(device, jobs).traversal for _ in range(4)]
    for gs, _, _ in jobs:
        gs.close()
    assert all(0 <= t <= highest for t in got), got
