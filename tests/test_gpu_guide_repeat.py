"""The guide's gradients are a function of the records and the parameters: the same records give the same
mean weight, hence the same bf16 operands and the same MLP gradients bit for bit, whichever warps finish
first.  The grid's gradients are atomic sums whose additions come in any order."""
import numpy as np
import pytest

from swpathtracer_b200 import abi
from test_gpu_guiding import _guide, _records

pytestmark = pytest.mark.gpu

# An entry is a sum of m 32-bit terms in any order: each of its m - 1 additions rounds by at most 2^-24 of
# the running sum.  The terms are of both signs, but those of one entry are few (2^18 records spread over
# the levels' cells, some hundreds in the coarsest): 16 roundings of the 2-norm.
GRID_TOL = 16 * 2.0 ** -24
# The loss adds the sums of at most 2 x 148 blocks of 4 warps, in any order.
LOSS_TOL = 2 * 148 * 4 * 2.0 ** -24


def _batch(n):
    r = _records(np.random.default_rng(41), n)
    r["weight"] = np.random.default_rng(42).exponential(1.0, n) ** 2   # the long tail of radiance estimates
    return r


@pytest.mark.parametrize("path,n", [(abi.GUIDE_TRAIN_TCGEN05, 1 << 18), (abi.GUIDE_TRAIN_TCGEN05, 100003),
                                    (abi.GUIDE_TRAIN_TCGEN05, 3), (abi.GUIDE_TRAIN_MMA_SYNC, 30011)])
def test_gradients_repeat(device, path, n):
    recs = _batch(n)
    g, _, _ = _guide(device, seed=13, train_path=path)
    grid, mlp, loss = g.gradients(recs)
    for _ in range(9):
        grid1, mlp1, loss1 = g.gradients(recs)
        assert mlp1.tobytes() == mlp.tobytes()
        assert np.linalg.norm(grid1 - grid) <= GRID_TOL * np.linalg.norm(grid)
        assert abs(loss1 - loss) <= LOSS_TOL * abs(loss)
    g.close()
