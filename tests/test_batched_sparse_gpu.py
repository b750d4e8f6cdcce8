"""Batches whose bricks hold few soup vertices, about 256 and many (the line
between working the soup out by vertex and out of records): the same soup,
normals and side outputs as each volume by itself, with the counts read and
without, and as the oracle's."""
import numpy as np
import pytest
import torch

from mc_util import assert_same_mesh, gpu_extract

pytestmark = pytest.mark.gpu

DIMS = [(64, 41, 33), (33, 9, 9), (65, 40, 30), (2, 2, 2), (72, 20, 17)]


def _volume(dims, share, seed):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    t = rng.integers(1, 30000, (nz, ny, nx)).astype(np.int16)
    t[rng.random(t.shape) < share] *= -1
    w = (rng.random(t.shape) > 0.0005).astype(np.int16)
    return np.stack([t, w], axis=-1)


@pytest.mark.parametrize("share", [0.0, 0.0005, 0.002, 0.005, 0.0055, 0.006, 0.02, 0.3])
def test_few_to_many(mcg, orc, share):
    host = [_volume(d, share, i) for i, d in enumerate(DIMS)]
    if share == 0.0:
        host[1][4, 4, 4, 0] = -5
    vols = [torch.from_numpy(v).cuda() for v in host]
    keys = ("soup", "normals", "vi2vox", "ver_voxel", "tri_cube")
    alone = [mcg.extract(v, 0.01, vi2vox=True, ver_voxel=True, tri_cube=True) for v in vols]
    for v in host:
        assert_same_mesh(gpu_extract(mcg, v, 0.01), orc.mc_extract(v, 0.01))
    read = mcg.extract_batched(vols, 0.01, vi2vox=True, ver_voxel=True, tri_cube=True)
    outs = [{k: torch.zeros_like(getattr(m, k)) for k in keys} for m in alone]
    mcg.extract_batched_into(vols, 0.01, outs, [m.num_vertices for m in alone], ctx=mcg.Context())
    torch.cuda.synchronize()
    for m, r, o in zip(alone, read, outs):
        for k in keys:
            assert torch.equal(getattr(r, k), getattr(m, k)) and torch.equal(o[k], getattr(m, k))
