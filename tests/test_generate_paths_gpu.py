"""Soup by records of crossed edges or vertex by vertex, whichever a volume's
soup vertices per brick choose: the same soup from a call whose counts the host
has read, from one call in which the device decides, from a second generate, and
from a captured graph replayed with volumes on either side.  Oracle: positions,
voxels and cubes bit for bit, normals too."""
import ctypes

import numpy as np
import pytest
import torch

from marching_cube_gb300 import _capi
from mc_util import assert_same_mesh, gpu_extract

pytestmark = pytest.mark.gpu

# share of negative voxels -> about 48500 times that many soup vertices a brick: the rules' ends are 256, 640 and 1300
SHARES = [0.0, 0.001, 0.01, 0.015, 0.0165, 0.02, 0.025, 0.0268, 0.03, 0.05, 0.1, 0.5]


def _volume(dims, share, seed=0):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    f = rng.uniform(0.01, 1.0, (nz, ny, nx)).astype(np.float32)
    f[rng.random(f.shape) < share] *= -1
    w = (rng.random(f.shape) > 0.0005).astype(np.float32)
    return np.stack([f, w], axis=-1)


def _one_call(mcg, ctx, vol, cell, n, normals=True):
    """mcg_mc_extract: the host has not read the counts"""
    nz, ny, nx, _ = vol.shape
    m = max(n, 3)
    o = {"soup": torch.zeros((m, 28), dtype=torch.uint8, device="cuda"),
         "normals": torch.zeros((m, 3), device="cuda") if normals else None,
         "vi2vox": torch.zeros((m, 3), dtype=torch.int32, device="cuda"),
         "ver_voxel": None, "tri_cube": torch.zeros((m // 3,), dtype=torch.int64, device="cuda")}
    cv = _capi.Volume(vol.data_ptr(), nx, ny, nz, 1, float(cell))
    mo = _capi.MeshOut(*(o[k].data_ptr() if o[k] is not None else None
                         for k in ("soup", "normals", "vi2vox", "ver_voxel", "tri_cube")), n)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ctx.check(mcg._lib.mcg_mc_extract(ctx.handle, ctypes.byref(cv), ctypes.byref(mo), s), "mcg_mc_extract")
    return o, (cv, mo)


def _same(o, mesh, n):
    assert torch.equal(o["soup"][:n], mesh.soup[:n]) and torch.equal(o["vi2vox"][:n], mesh.vi2vox[:n])
    assert torch.equal(o["tri_cube"][:n // 3], mesh.tri_cube[:n // 3])
    if o["normals"] is not None:
        assert torch.equal(o["normals"][:n], mesh.normals[:n])


@pytest.mark.parametrize("dims", [(64, 41, 33), (65, 40, 30)])
@pytest.mark.parametrize("share", SHARES)
def test_both_ways(mcg, orc, dims, share):
    vol = _volume(dims, share)
    assert_same_mesh(gpu_extract(mcg, vol, 0.01), orc.mc_extract(vol, 0.01))
    v = torch.from_numpy(vol).cuda()
    mesh = mcg.extract(v, 0.01, vi2vox=True, tri_cube=True)
    n = mesh.num_vertices
    ctx = mcg.Context()
    for normals in (True, False):
        o, (cv, mo) = _one_call(mcg, ctx, v, 0.01, n, normals)
        # a second generate after the same count phase, before and after the counts are read
        for _ in range(2):
            o["soup"].zero_()
            s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
            ctx.check(mcg._lib.mcg_mc_generate(ctx.handle, ctypes.byref(cv), ctypes.byref(mo), s), "mcg_mc_generate")
            c = mcg.counts(ctx)
            assert c["vertices"] == n and c["status"] == 0
            _same(o, mesh, n)


def test_graph_of_either(mcg):
    dims = (64, 41, 33)
    vols = [torch.from_numpy(_volume(dims, p, seed=i)).cuda() for i, p in enumerate((0.02, 0.001, 0.022, 0.1, 0.0, 0.02))]
    meshes = [mcg.extract(v, 0.01, vi2vox=True, tri_cube=True) for v in vols]
    n = max(m.num_vertices for m in meshes)
    v, ctx = vols[0].clone(), mcg.Context()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        _one_call(mcg, ctx, v, 0.01, n)
        st.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            o, _ = _one_call(mcg, ctx, v, 0.01, n)
    for src, mesh in zip(vols, meshes):
        v.copy_(src)
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert mcg.counts(ctx)["vertices"] == mesh.num_vertices
        _same(o, mesh, mesh.num_vertices)


@pytest.mark.parametrize("dims", [(64, 41, 33), (65, 40, 30), (72, 20, 17)])
@pytest.mark.parametrize("share", [0.0005, 0.002, 0.005, 0.0053, 0.006, 0.02])
def test_short_volumes(mcg, orc, dims, share):
    """256 soup vertices a brick, either side; the host has read the counts or not."""
    v = _volume(dims, share)
    vol = np.stack([(v[..., 0] * 30000).astype(np.int16), v[..., 1].astype(np.int16)], axis=-1)
    vol[..., 0][(vol[..., 0] == 0)] = 7
    o = orc.mc_extract(vol, 0.01)
    assert_same_mesh(gpu_extract(mcg, vol, 0.01), o)
    t = torch.from_numpy(vol).cuda()
    mesh = mcg.extract(t, 0.01, vi2vox=True, ver_voxel=True, tri_cube=True)
    out = {k: torch.zeros_like(getattr(mesh, k)) for k in ("soup", "normals", "vi2vox", "ver_voxel", "tri_cube")}
    mcg.extract_into(t, 0.01, out, mesh.num_vertices, ctx=mcg.Context())
    assert all(torch.equal(out[k], getattr(mesh, k)) for k in out)
    for keep in (("soup",), ("normals",), ("soup", "normals", "tri_cube")):
        part = mcg.extract(t, 0.01, **{k: k in keep for k in out})
        assert all(torch.equal(getattr(part, k), getattr(mesh, k)) for k in keep)
