"""Gradients of small and ragged batches, whose records are copied in and encoded in up to eight parts,
against the warp-level training path, which takes them in one piece."""
import numpy as np
import pytest

from swpathtracer_b200 import abi
from test_gpu_guiding import _guide, _records

pytestmark = pytest.mark.gpu

# Both paths round the same operands to bf16 and accumulate in 32 bits in different orders: an activation
# may land on the neighbouring bf16 value (2^-8 apart) in each of the five layers.
TOL = 5 * 2.0 ** -8


@pytest.mark.parametrize("n", [1, 2, 129, 1023, (1 << 16) - 1, (1 << 16) + 1, (1 << 17) + 3])
def test_parts_match_one_piece(device, n):
    recs = [_records(np.random.default_rng(seed), n) for seed in (31, 32)]
    out = {}
    for path in (abi.GUIDE_TRAIN_TCGEN05, abi.GUIDE_TRAIN_MMA_SYNC):
        g, _, _ = _guide(device, seed=9, train_path=path)
        # a second batch follows at once: it must not see the first one's records or sums
        out[path] = [g.gradients(r) for r in recs]
        g.close()
    for (ga, ma, la), (gb, mb, lb) in zip(out[abi.GUIDE_TRAIN_TCGEN05], out[abi.GUIDE_TRAIN_MMA_SYNC]):
        assert abs(la - lb) <= TOL * max(abs(lb), 1.0)
        assert np.linalg.norm(ma - mb) <= TOL * np.linalg.norm(mb)
        assert np.linalg.norm(ga - gb) <= TOL * np.linalg.norm(gb)
