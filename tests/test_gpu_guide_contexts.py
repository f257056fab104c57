"""A guide's gradients and training steps may come by another context than the guide's own: they run on the
caller's stream, and the calls follow one another as if they all came by one context."""
import numpy as np
import pytest
import torch

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi
from test_gpu_guide_repeat import GRID_TOL
from test_gpu_guiding import _records

pytestmark = pytest.mark.gpu


def _pinned(recs):
    return torch.from_numpy(recs.view(np.uint8).copy()).pin_memory().numpy().view(abi.GUIDE_RECORD_DTYPE)


@pytest.mark.parametrize("path", [abi.GUIDE_TRAIN_TCGEN05, abi.GUIDE_TRAIN_MMA_SYNC])
def test_calls_by_two_contexts(device, path):
    n = 1 << 17
    recs = [_pinned(_records(np.random.default_rng(70 + k), n)) for k in range(3)]
    other = spt.Device(0)
    out = []
    for by in ([device] * 5, [other, device, other, device, other]):
        g = spt.Guide(device, spt.guide_config(batch=n, cache_res=4, seed=5, train_path=path))
        start, _ = g.get_params()
        grads = []
        for k, dev in enumerate(by[:4]):
            g.dev = dev   # the context the next call comes by
            grads.append(g.gradients(recs[k % 3]))
        g.dev = by[4]
        g.train(recs[2])
        grid, mlp = g.get_params()
        g.dev = device
        g.close()
        out.append((grads, grid != start, mlp))
    (grads_a, moved_a, mlp_a), (grads_b, moved_b, mlp_b) = out
    for (ga, ma, _), (gb, mb, _) in zip(grads_a, grads_b):
        assert ma.tobytes() == mb.tobytes()
        assert np.linalg.norm(ga - gb) <= GRID_TOL * np.linalg.norm(ga)
    assert mlp_a.tobytes() == mlp_b.tobytes()
    # the step moved the entries of its own batch, none of the gradient calls' before it (a sum may cancel
    # to exactly zero in one order of its additions and not in another)
    assert np.count_nonzero(moved_a != moved_b) <= 1e-5 * np.count_nonzero(moved_a)
    other.close()
