"""A guide's first gradient call or training step of up to its configured batch allocates no device memory."""
import numpy as np
import pytest
import torch

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi
from test_gpu_guiding import _records

pytestmark = pytest.mark.gpu

BATCH = 1 << 17


@pytest.mark.parametrize("path", [abi.GUIDE_TRAIN_TCGEN05, abi.GUIDE_TRAIN_MMA_SYNC])
@pytest.mark.parametrize("call,n", [("gradients", BATCH), ("gradients", 1), ("train", BATCH)])
def test_first_call_allocates_nothing(path, call, n):
    dev = spt.Device(0)   # a context of its own: no scratch buffer that an earlier call has grown
    warm = spt.Guide(dev, spt.guide_config(batch=1024, cache_res=4, train_path=path))
    recs = _records(np.random.default_rng(61), n)
    getattr(warm, call)(recs[:1024])   # the kernels' code is loaded on first use
    warm.close()
    g = spt.Guide(dev, spt.guide_config(batch=BATCH, cache_res=4, train_path=path))
    torch.cuda.synchronize()
    before, _ = torch.cuda.mem_get_info()
    getattr(g, call)(recs)
    torch.cuda.synchronize()
    after, _ = torch.cuda.mem_get_info()
    assert after == before
    g.close()
    dev.close()


def test_batches_beyond_the_configured_one_still_run(device):
    g = spt.Guide(device, spt.guide_config(batch=256, cache_res=4, seed=7))
    ref = spt.Guide(device, spt.guide_config(batch=4096, cache_res=4, seed=7))
    recs = _records(np.random.default_rng(62), 4001)
    (_, ma, _), (_, mb, _) = g.gradients(recs), ref.gradients(recs)
    assert ma.tobytes() == mb.tobytes()
    g.close()
    ref.close()
