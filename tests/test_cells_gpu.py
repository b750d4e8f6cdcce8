"""Cells and sides for which positions leave the nodes that they lie between:
coordinates that overflow (an infinite cell, one that overflows at some voxel on,
where the second end of an edge may alone be infinite), subnormal cells, sides
beyond 2^22 voxels.  Voxel and normal of every vertex are those of its position
(a conversion of NaN gives 0, of an infinite one the largest int), whichever
launch works them out.  Positions and whatever is finite: the oracle, bit for
bit; the rest by numpy, and by the launch that takes normals at given positions."""
import ctypes

import numpy as np
import pytest
import torch

from marching_cube_gb300 import _capi
from mc_util import VERTEX_DTYPE, assert_same_mesh, gpu_extract

pytestmark = pytest.mark.gpu

KEYS = ("soup", "normals", "vi2vox", "ver_voxel", "tri_cube")


def _volume(dims, p, seed=3):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    t = rng.integers(0, 32767, (nz, ny, nx))
    t[rng.random(t.shape) < p] *= -1
    w = rng.integers(1, 60000, t.shape).astype(np.uint16)
    return np.stack([t.astype(np.int16), w.view(np.int16)], axis=-1)


def _whole(x):
    out = np.zeros(x.shape, np.int64)
    fine = ~np.isnan(x)
    out[fine] = np.clip(x[fine].astype(np.float64), -2.0**31, 2.0**31 - 1).astype(np.int64)
    return out


def _fused(mcg, vol, cell, n, mode):
    ctx = mcg.Context()
    ctx.set_config(fused=mode)
    nz, ny, nx, _ = vol.shape
    o = {"soup": torch.zeros((n, 28), dtype=torch.uint8, device="cuda"),
         "normals": torch.zeros((n, 3), dtype=torch.float32, device="cuda"),
         "vi2vox": torch.zeros((n, 3), dtype=torch.int32, device="cuda"),
         "ver_voxel": torch.zeros((nx * ny * nz,), dtype=torch.int16, device="cuda"),
         "tri_cube": torch.zeros((n // 3,), dtype=torch.int64, device="cuda")}
    cv = _capi.Volume(vol.data_ptr(), nx, ny, nz, 0, float(cell))
    mo = _capi.MeshOut(*(o[k].data_ptr() for k in KEYS), n)
    ctx.check(mcg._lib.mcg_mc_extract(ctx.handle, ctypes.byref(cv), ctypes.byref(mo),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "mcg_mc_extract")
    assert mcg.counts(ctx)["vertices"] == n
    return o


def _bytes(t):
    return t.contiguous().view(torch.uint8).cpu()


def _check(mcg, orc, vol, cell):
    v = torch.from_numpy(vol).cuda()
    kw = dict(soup=True, normals=True, vi2vox=True, ver_voxel=True, tri_cube=True)
    mesh = mcg.extract(v, cell, **kw)
    n = mesh.num_vertices
    assert n > 0
    g = mesh.soup.cpu().numpy().reshape(-1).view(VERTEX_DTYPE)
    order = np.argsort(mesh.tri_cube.cpu().numpy(), kind="stable")
    idx = (order[:, None] * 3 + np.arange(3)).reshape(-1)
    want = orc.mc_extract(vol, cell)["soup"]["pos"]
    got = g["pos"][idx]
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan) and np.array_equal(got[~nan], want[~nan])
    # the voxel, its distance and weight
    with np.errstate(all="ignore"):
        pf = g["pos"] / np.float32(cell)
        vox = _whole(np.floor(pf - np.float32(0.5)))
    nz, ny, nx, _ = vol.shape
    assert np.array_equal(g["vox"], vox) and np.array_equal(mesh.vi2vox.cpu().numpy(), vox)
    li = (vox[:, 2] * ny + vox[:, 1]) * nx + vox[:, 0]
    there = (li >= 0) & (li < nx * ny * nz)
    flat = vol.reshape(-1, 2)
    at = flat[np.where(there, li, 0)] * there[:, None].astype(np.int16)
    assert np.array_equal(g["tsdf"], at[:, 0]) and np.array_equal(g["w"], at[:, 1])
    written = np.zeros(nx * ny * nz, np.int16)
    written[li[there]] = flat[li[there], 0]
    assert np.array_equal(mesh.ver_voxel.cpu().numpy().reshape(-1), written)
    # the normal
    normals = mcg.extract_surface_normals(v, cell, mesh.soup)
    nan = torch.isnan(normals)
    assert torch.equal(torch.isnan(mesh.normals), nan) and torch.equal(mesh.normals[~nan], normals[~nan])
    # the other launches
    others = [mcg.extract_batched([v, v], [cell, cell], **kw)[1]]
    others = [{k: getattr(o, k) for k in KEYS} for o in others] + [_fused(mcg, v, cell, n, m) for m in (1, 2)]
    for o in others:
        for k in KEYS:
            a, b = getattr(mesh, k), o[k]
            if k == "normals":
                assert torch.equal(torch.isnan(b), nan) and torch.equal(a[~nan], b[~nan])
            elif k == "soup":
                pa, pb = _bytes(a).numpy().view(VERTEX_DTYPE).reshape(-1), _bytes(b).numpy().view(VERTEX_DTYPE).reshape(-1)
                assert np.array_equal(pa["pos"], pb["pos"], equal_nan=True)
                assert all(np.array_equal(pa[f], pb[f]) for f in ("vox", "tsdf", "w"))
            else:
                assert torch.equal(a.reshape(-1), b.reshape(-1)), k


@pytest.mark.parametrize("p", [0.02, 0.5])
@pytest.mark.parametrize("dims", [(70, 19, 17), (36, 40, 28), (52, 12, 40)])
@pytest.mark.parametrize("cell", [float("inf"), 1.7e37, 2.2e37, 1e38, 3e38, 1.4e-45, 2.8e-45, 1e-38])
def test_cells(mcg, orc, cell, dims, p):
    _check(mcg, orc, _volume(dims, p), cell)


@pytest.mark.parametrize("cell", [float("inf"), 1.7e37, 1.4e-45])
def test_float_volume(mcg, orc, cell):
    v = _volume((52, 20, 24), 0.05)
    vol = np.stack([v[..., 0] / np.float32(32766), (v[..., 1] != 0).astype(np.float32)], axis=-1).astype(np.float32)
    g = gpu_extract(mcg, vol, cell, canonical=False)
    o = gpu_extract(mcg, v, cell, canonical=False)  # 16-bit distances: the same unpacked values
    assert np.array_equal(g["tri_cube"], o["tri_cube"]) and np.array_equal(g["vi2vox"], o["vi2vox"])
    assert np.array_equal(g["soup"]["pos"], o["soup"]["pos"], equal_nan=True)
    # (distances of floats have no bounds, so a normal next to +-32766 is not zero here)
    f = torch.from_numpy(vol).cuda()
    mesh = mcg.extract(f, cell)
    assert np.array_equal(mesh.normals.cpu().numpy(), g["normals"], equal_nan=True)
    want = mcg.extract_surface_normals(f, cell, mesh.soup).cpu().numpy()
    assert np.array_equal(g["normals"], want, equal_nan=True)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("side", [(1 << 21) + 40, 6000000])
def test_long_sides(mcg, orc, side, axis):
    long = 20000
    dims = [2, 2, 2]
    dims[axis] = long
    tail = _volume(dims, 0.2)
    shape = [2, 2, 2, 2]
    shape[2 - axis] = side
    vol = np.full(shape, 1000, np.int16)
    vol[tuple(slice(side - long, side) if a == 2 - axis else slice(None) for a in range(3))] = tail
    assert_same_mesh(gpu_extract(mcg, vol, 0.0037), orc.mc_extract(vol, 0.0037))
