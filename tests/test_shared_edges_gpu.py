"""The soup from records of crossed edges: bricks around what is taken in
hand at a time (1600 soup vertices, 640 records, 768 occupied cubes) -- none,
few, exactly one plane of 1536, several planes in every direction (several
groups of layers), more than fit (each soup vertex for itself) -- one brick and
ragged neighbours, a cell whose reciprocal is not used (significand all ones)
and one out of its range, outputs that end inside a brick, subsets of the
outputs.  Oracle: every output bit for bit."""
import numpy as np
import pytest
import torch

from mc_util import assert_same_mesh, gpu_extract

pytestmark = pytest.mark.gpu

KINDS = ["px3", "py2", "pz2", "pz4", "pz8", "py8", "pd5", "pd9", "pd14", "r0.0", "r0.003", "r0.01", "r0.03", "r0.1", "r0.5"]
CELLS = [0.0037, float(np.uint32(0x3c7fffff).view(np.float32)), 1e-30, 3.0]


def _volume(kind, dims, seed=1):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    if kind[0] == "p":
        a = {"x": x, "y": y, "z": z, "d": x + y + z}[kind[1]]
        s = np.where((a // int(kind[2:])) % 2, 1, -1)
    else:
        s = np.where(rng.random(x.shape) < float(kind[1:]), -1, 1)
    t = s * rng.integers(1, 32767, x.shape)
    t[(t > 0) & (rng.random(x.shape) < 0.02)] = 0
    w = rng.integers(1, 60000, x.shape).astype(np.uint16)
    w[rng.random(x.shape) < 0.01] = 0
    return np.stack([t.astype(np.int16), w.view(np.int16)], axis=-1)


@pytest.mark.parametrize("dims", [(33, 9, 9), (36, 12, 12), (70, 19, 17)])
@pytest.mark.parametrize("kind", KINDS)
def test_bricks(mcg, orc, kind, dims):
    vol = _volume(kind, dims)
    cell = CELLS[len(kind) % 4]
    assert_same_mesh(gpu_extract(mcg, vol, cell), orc.mc_extract(vol, cell))


@pytest.mark.parametrize("cell", CELLS)
def test_cells(mcg, orc, cell):
    vol = _volume("r0.03", (50, 21, 23))
    assert_same_mesh(gpu_extract(mcg, vol, cell), orc.mc_extract(vol, cell))


@pytest.mark.parametrize("kind", ["pd9", "pz4", "r0.01"])
def test_float_volume(mcg, orc, kind):
    v = _volume(kind, (40, 17, 20))
    vol = np.stack([v[..., 0] / np.float32(32766), (v[..., 1] != 0).astype(np.float32)], axis=-1).astype(np.float32)
    vol[3, 4, 5, 0], vol[3, 4, 6, 0] = -1e-15, 0.0  # an interpolation at 0 / 0 when the edge runs down
    g, o = gpu_extract(mcg, vol, 0.01), orc.mc_extract(vol, 0.01)
    # where the position is not finite its voxel is a conversion that C leaves
    # undefined, and ver_voxel may have been written there
    fine = np.isfinite(o["soup"]["pos"]).all(axis=1)
    assert np.array_equal(np.isfinite(g["soup"]["pos"]).all(axis=1), fine)
    assert np.array_equal(g["tri_cube"], o["tri_cube"])
    for k in ("soup", "normals", "vi2vox"):
        assert np.array_equal(np.ascontiguousarray(g[k][fine]).view(np.uint8), np.ascontiguousarray(o[k][fine]).view(np.uint8))


@pytest.mark.parametrize("keep", [("soup",), ("normals",), ("soup", "vi2vox"), ("normals", "tri_cube"), ("soup", "ver_voxel")])
def test_capacity_and_subsets(mcg, keep):
    vol = torch.from_numpy(_volume("pd9", (70, 19, 17))).cuda()
    whole = mcg.extract(vol, 0.01, soup=True, normals=True, vi2vox=True, ver_voxel=True, tri_cube=True)
    n = whole.num_vertices
    parts = {"soup": whole.soup, "normals": whole.normals, "vi2vox": whole.vi2vox, "tri_cube": whole.tri_cube}
    for cap in (n, n - 1, n - 2000, 1537, 1):
        out = {k: torch.full_like(parts[k], 7) for k in keep if k != "ver_voxel"}
        if "ver_voxel" in keep:
            out["ver_voxel"] = torch.empty_like(whole.ver_voxel)
        ctx = mcg.extract_into(vol, 0.01, out, cap)
        c = mcg.counts(ctx)
        assert c["vertices"] == n
        for k in keep:
            if k == "ver_voxel":
                if cap == n:
                    assert torch.equal(out[k], whole.ver_voxel)
                continue
            m = cap // 3 if k == "tri_cube" else cap
            assert torch.equal(out[k][:m], parts[k][:m])
            assert bool((out[k][m:] == 7).all())


@pytest.mark.parametrize("upwards", [True, False])
@pytest.mark.parametrize("n", [50, 63, 64, 65, 66, 67, 68, 90])
def test_isolated_voxels(mcg, orc, n, upwards):
    """Isolated negative voxels, 24 soup vertices and 10 records each, around the
    64 whose records fit, in the lower or the upper layers of the brick."""
    at = [(z, y, x) for z in (1, 4, 7) for y in (1, 4, 7) for x in range(2, 32, 3)]
    vol = np.full((9, 9, 33, 2), 1000, np.int16)
    for z, y, x in (at if upwards else at[::-1])[:n]:
        vol[z, y, x, 0] = -700
    o = orc.mc_extract(vol, 0.01)
    assert len(o["soup"]) == 24 * n
    assert_same_mesh(gpu_extract(mcg, vol, 0.01), o)
