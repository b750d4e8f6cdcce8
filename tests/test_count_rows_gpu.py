"""The count pass by rows (volumes TMA cannot describe, and batches) at its
edges: bricks that fill their 33 x 9 x 9 voxels exactly, end one short or one
past, sides of two voxels, distances of one sign but for the 33rd column or a
corner of the last plane, bases at every voxel offset, slabs; counts and soup
against the oracle."""
import numpy as np
import pytest
import torch

from marching_cube_gb300 import synthetic
from mc_util import assert_same_mesh, mesh_arrays

pytestmark = pytest.mark.gpu

DIMS = [(2, 2, 2), (33, 9, 9), (34, 10, 10), (32, 8, 8), (65, 17, 17), (66, 18, 18), (35, 2, 40), (3, 41, 2), (97, 25, 33)]


def _extract(mcg, view, cell, **kw):
    m = mcg.extract(view, cell, soup=True, normals=True, vi2vox=True, ver_voxel=True, tri_cube=True, **kw)
    torch.cuda.synchronize()
    return mesh_arrays(m)


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("vtype", [torch.int16, torch.float32])
def test_random(mcg, orc, dims, vtype):
    nx, ny, nz = dims
    vol = synthetic.random_volume((nz, ny, nx), seed=nx + ny, p_zero_weight=0.02)
    if vtype == torch.float32:
        vol = np.stack([vol[..., 0] / np.float32(32766), (vol[..., 1] != 0).astype(np.float32)], axis=-1).astype(np.float32)
    n = nx * ny * nz
    for offset in (0, 1, 3):
        buf = torch.zeros((n + 8, 2), dtype=vtype, device="cuda")
        view = buf[offset:offset + n].view(nz, ny, nx, 2)
        view.copy_(torch.from_numpy(vol))
        assert_same_mesh(_extract(mcg, view, 0.01), orc.mc_extract(vol, 0.01))


@pytest.mark.parametrize("where", ["column", "corner", "first", "none"])
@pytest.mark.parametrize("negative", [False, True])
def test_one_voxel(mcg, orc, where, negative):
    nx, ny, nz = 33, 9, 9
    vol = np.full((nz, ny, nx, 2), 9, np.int16)
    vol[..., 0] = -500 if negative else 500
    at = {"column": (4, 4, 32), "corner": (8, 8, 32), "first": (0, 0, 0), "none": None}[where]
    if at:
        vol[at + (0,)] = 500 if negative else -500
    g = _extract(mcg, torch.from_numpy(vol).cuda(), 0.01)
    o = orc.mc_extract(vol, 0.01)
    assert len(g["soup"]) == (0 if at is None else len(o["soup"])) and (at is None or len(g["soup"]) > 0)
    assert_same_mesh(g, o)


def test_batch_and_slabs(mcg, orc):
    vols = [synthetic.random_volume((nz, ny, nx), seed=7 * i, p_zero_weight=0.02) for i, (nx, ny, nz) in enumerate(DIMS)]
    vols += [synthetic.random_volume((16, 16, 64), seed=5), synthetic.random_volume((40, 24, 36), seed=6)]
    t = [torch.from_numpy(v).cuda() for v in vols]
    for v, m in zip(vols, mcg.extract_batched(t, 0.01, vi2vox=True, ver_voxel=True, tri_cube=True)):
        torch.cuda.synchronize()
        assert_same_mesh(mesh_arrays(m), orc.mc_extract(v, 0.01))
    whole = mcg.extract(t[8], 0.01)
    parts = [mcg.extract_slab(t[8], 0.01, z0, z1) for z0, z1 in ((0, 8), (8, 24), (24, 32))]
    torch.cuda.synchronize()
    assert torch.equal(torch.cat([p.soup for p in parts]), whole.soup)
