"""Parameters set at any time reach every copy of them that a later call reads: a guide that has already
computed gradients or taken a step, and then gets other parameters, is the guide created with them."""
import numpy as np
import pytest

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi
from test_gpu_guide_repeat import GRID_TOL
from test_gpu_guiding import _guide, _records

pytestmark = pytest.mark.gpu


def _params(seed):
    g = np.random.default_rng(seed)
    return (g.uniform(-0.5, 0.5, abi.GUIDE_GRID_PARAMS).astype(np.float32),
            (0.2 * g.standard_normal(abi.GUIDE_MLP_PARAMS)).astype(np.float32))


@pytest.mark.parametrize("path", [abi.GUIDE_TRAIN_TCGEN05, abi.GUIDE_TRAIN_MMA_SYNC])
@pytest.mark.parametrize("before", ["nothing", "gradients", "train"])
@pytest.mark.parametrize("which", ["both", "mlp"])
def test_set_params_reaches_the_gradients(device, path, before, which):
    n = 2085
    recs = _records(np.random.default_rng(51), n)
    grid, mlp = _params(52)
    used, old_grid, _ = _guide(device, seed=14, train_path=path)
    if before == "gradients":
        used.gradients(recs)
    if before == "train":
        used.train(recs)
        old_grid, _ = used.get_params()
    fresh = spt.Guide(device, spt.guide_config(seed=15, train_path=path))
    used.set_params(grid=grid if which == "both" else None, mlp=mlp)
    fresh.set_params(grid=grid if which == "both" else old_grid, mlp=mlp)
    (ga, ma, _), (gb, mb, _) = used.gradients(recs), fresh.gradients(recs)
    assert ma.tobytes() == mb.tobytes()
    assert np.linalg.norm(ga - gb) <= GRID_TOL * np.linalg.norm(gb)
    used.close()
    fresh.close()
