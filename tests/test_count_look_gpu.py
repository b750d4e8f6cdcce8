"""The count pass by rows where a warp takes several bricks and looks at the signs
of a short2 brick first, or not, by the brick before: regions of one sign, of
noise, and of single voxels at the edges of bricks, next to one another; one
volume TMA cannot describe, and batches.  Soup and counts against the oracle."""
import numpy as np
import pytest
import torch

from mc_util import assert_same_mesh, mesh_arrays

pytestmark = pytest.mark.gpu


def _volume(dims, seed):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    t = rng.integers(1, 32766, (nz, ny, nx)).astype(np.int16)
    t[nz // 5: nz // 4] *= -1  # a slab behind a surface
    t[nz // 2:, :, : nx // 5][rng.random((nz - nz // 2, ny, nx // 5)) < 0.2] *= -1
    # single voxels where bricks (32 x 8 x 8 cubes) end and begin
    n = 300
    z, y, x = (np.minimum(rng.integers(0, s // b + 1, n) * b + rng.integers(-1, 2, n), s - 1).clip(0)
               for s, b in ((nz, 8), (ny, 8), (nx, 32)))
    t[z, y, x] = -7
    t[-1, -1, -1] = t[0, 0, 0] = -3
    w = (rng.random((nz, ny, nx)) > 0.001).astype(np.int16)
    return np.stack([t, w], axis=-1)


def test_one_volume(mcg, orc):
    vol = _volume((323, 171, 190), 1)  # 11 x 22 x 24 bricks; 3648 warps (152 SMs, 3 CTAs of 8)
    m = mcg.extract(torch.from_numpy(vol).cuda(), 0.01, vi2vox=True, ver_voxel=True, tri_cube=True)
    torch.cuda.synchronize()
    assert_same_mesh(mesh_arrays(m), orc.mc_extract(vol, 0.01))


def test_batch(mcg, orc):
    # 19180 bricks, one after another; and so many that four are drawn at a time (from 58368 on)
    for repeat in (1, 6):
        vols = [_volume(d, 2 + i) for i, d in enumerate([(323, 171, 190), (64, 100, 100), (2, 300, 301), (160, 160, 160)])]
        dev = [torch.from_numpy(v).cuda() for v in vols]
        dev += dev * (2 * repeat - 1)
        meshes = mcg.extract_batched(dev, 0.01, vi2vox=True, ver_voxel=True, tri_cube=True)
        torch.cuda.synchronize()
        for i, v in enumerate(vols):
            assert_same_mesh(mesh_arrays(meshes[i]), orc.mc_extract(v, 0.01))
        for i, m in enumerate(meshes):
            assert torch.equal(m.soup, meshes[i % 4].soup) and torch.equal(m.normals, meshes[i % 4].normals)
