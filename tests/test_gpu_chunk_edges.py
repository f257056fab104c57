"""Queries from page-locked host memory around the pipeline's chunk of 2^19 rays, and guide gradients around
the edges of the parts that their records are copied in."""
import numpy as np
import pytest
import torch

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi, scenes
from test_gpu_guide_parts import TOL
from test_gpu_guiding import _guide, _records

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh(device):
    gs = spt.GpuScene(device, scenes.displaced_mesh_scene(5).build())
    yield gs
    gs.close()


@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19, (1 << 19) + 1, 1 << 20, (1 << 20) + 1, (1 << 21) + 77])
@pytest.mark.parametrize("floats", [8, 6])
def test_host_queries_around_the_chunk(mesh, n, floats):
    rays = scenes.incoherent_rays(n, seed=n & 0xFF, half_extent=1.5)
    d_rays = torch.from_numpy(rays).cuda()
    d_hits = torch.empty((n, 4), dtype=torch.int32, device="cuda")
    mesh.intersect_device(d_rays.data_ptr(), n, d_hits.data_ptr(), 0)
    torch.cuda.synchronize()
    if floats == 6:
        rays = np.ascontiguousarray(np.concatenate([rays[:, 0:3], rays[:, 4:7]], axis=1))
    h_rays = torch.from_numpy(rays).pin_memory()
    # one record more than the batch: nothing is written behind its end
    h_hits = torch.full((n + 1, 4), 7, dtype=torch.int32).pin_memory()
    out = h_hits.numpy().view(abi.HIT_DTYPE).reshape(n + 1)
    mesh.intersect(h_rays.numpy(), out=out[:n])
    assert torch.equal(h_hits[:n], d_hits.cpu())
    assert bool((h_hits[n] == 7).all())


@pytest.mark.parametrize("n,parts", [((1 << 16) + 1, 2), ((1 << 17) + 3, 4), ((1 << 18) + 3, 8), ((1 << 18) + 1029, 8)])
@pytest.mark.parametrize("where", ["starts", "ends", "last"])
def test_records_at_the_edges_of_the_parts_count(device, n, parts, where):
    """All the weight on a few records beside the parts' edges, so that the gradient is theirs alone: a part
    or a tile left out, taken twice or read before it has arrived is an error of the size of the gradient."""
    recs = [_records(np.random.default_rng(seed), n) for seed in (81, 82)]
    per = (n + parts - 1) // parts
    for r in recs:
        w = np.zeros(n, np.float32)
        if where == "last":
            w[-1] = 1.0
        for p in range(parts):
            first, last = p * per, min(n, (p + 1) * per)
            if where == "starts":
                w[first:first + 3] = 1.0
            if where == "ends":
                w[last - 3:last] = 1.0
        r["weight"] = w
    out = {}
    for path in (abi.GUIDE_TRAIN_TCGEN05, abi.GUIDE_TRAIN_MMA_SYNC):
        g, _, _ = _guide(device, seed=9, train_path=path)
        out[path] = [g.gradients(r) for r in recs]
        g.close()
    for (ga, ma, la), (gb, mb, lb) in zip(out[abi.GUIDE_TRAIN_TCGEN05], out[abi.GUIDE_TRAIN_MMA_SYNC]):
        assert abs(la - lb) <= TOL * max(abs(lb), 1.0)
        assert np.linalg.norm(ma - mb) <= TOL * np.linalg.norm(mb)
        assert np.linalg.norm(ga - gb) <= TOL * np.linalg.norm(gb)
