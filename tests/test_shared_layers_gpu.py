"""Bricks whose edge records are taken some layers of cubes at a time: a layer with
more soup vertices than are mapped at once (1599; it goes out in parts), layers
whose records (640) end before their soup vertices do, such layers first, in the
middle and last with empty ones around, and a layer whose own records do not
fit.  One brick and ragged neighbours; oracle: every output bit for bit."""
import numpy as np
import pytest
import torch

from mc_util import assert_same_mesh, gpu_extract

pytestmark = pytest.mark.gpu


def _volume(dims, at, flips, sparse, seed=1):
    """Negative below a sheet just above voxel plane `at` (from either side), the
    two planes at the sheet flipped with probability `flips`, and voxels of the
    whole volume with probability `sparse`."""
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    neg = np.zeros((nz, ny, nx), bool)
    if at is not None:
        neg[:at + 1] = True
        neg[at:at + 2] ^= rng.random((2, ny, nx)) < flips
    neg ^= rng.random(neg.shape) < sparse
    t = rng.integers(1, 32767, neg.shape)
    t[neg] *= -1
    return np.stack([t.astype(np.int16), np.ones(neg.shape, np.int16)], axis=-1)


def _layers(o, dims):
    nx, ny, _ = dims
    return np.bincount(o["tri_cube"] // (nx * ny), minlength=8)[:8] * 3


@pytest.mark.parametrize("dims", [(33, 9, 9), (70, 19, 17), (72, 20, 17)])
@pytest.mark.parametrize("at", [0, 3, 7])
@pytest.mark.parametrize("flips,sparse", [(0.02, 0.0), (0.08, 0.0), (0.25, 0.0), (0.02, 0.002), (0.08, 0.01), (0.5, 0.0)])
def test_layers(mcg, orc, dims, at, flips, sparse):
    vol = _volume(dims, at, flips, sparse)
    o = orc.mc_extract(vol, 0.01)
    if dims[0] == 33:
        layers = _layers(o, dims)
        assert layers.max() > 1599 and layers.sum() < 1 << 13
    assert_same_mesh(gpu_extract(mcg, vol, 0.01), o)


@pytest.mark.parametrize("dims", [(33, 9, 9), (70, 19, 17), (72, 20, 17)])
@pytest.mark.parametrize("sparse", [0.02, 0.025, 0.03, 0.04, 0.05, 0.06])
def test_records_end_first(mcg, orc, dims, sparse):
    vol = _volume(dims, None, 0.0, sparse)
    assert_same_mesh(gpu_extract(mcg, vol, 0.01), orc.mc_extract(vol, 0.01))


@pytest.mark.parametrize("sparse", [0.002, 0.02, 0.04])
def test_other_outputs(mcg, sparse):
    """Capacities that end inside a part, batches and float2 volumes."""
    vol = _volume((70, 19, 17), 3, 0.08, sparse)
    v = torch.from_numpy(vol).cuda()
    kw = dict(soup=True, normals=True, vi2vox=True, ver_voxel=True, tri_cube=True)
    whole = mcg.extract(v, 0.01, **kw)
    both = mcg.extract_batched([v, v], [0.01, 0.01], **kw)
    for m in both:
        assert all(torch.equal(getattr(m, k), getattr(whole, k)) for k in kw)
    # (numpy's division is IEEE's, as the 16-bit distances' is; torch multiplies by a reciprocal)
    f = np.stack([vol[..., 0] / np.float32(32766), vol[..., 1].astype(np.float32)], axis=-1).astype(np.float32)
    mesh = mcg.extract(torch.from_numpy(f).cuda(), 0.01, vi2vox=True, tri_cube=True)
    assert torch.equal(mesh.positions, whole.positions) and torch.equal(mesh.vi2vox, whole.vi2vox)
    assert torch.equal(mesh.tri_cube, whole.tri_cube)
    n = whole.num_vertices
    for cap in (n - 1, n // 2, 1600):
        out = {"soup": torch.full_like(whole.soup, 7), "tri_cube": torch.full_like(whole.tri_cube, 7)}
        mcg.extract_into(v, 0.01, out, cap)
        assert torch.equal(out["soup"][:cap], whole.soup[:cap]) and bool((out["soup"][cap:] == 7).all())
        assert torch.equal(out["tri_cube"][:cap // 3], whole.tri_cube[:cap // 3])
        assert bool((out["tri_cube"][cap // 3:] == 7).all())
