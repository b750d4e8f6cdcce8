"""The ray march fetches a ray's next samples together: volumes and images
at the edges of that, against the oracle's one-by-one march bit for bit --
no free space at all (random distances), free space that ends within a batch,
rays that leave the volume within one, thin bands crossed without a hit,
odd images and the smallest volume."""
import numpy as np
import pytest
import torch

from marching_cube_gb300 import synthetic

pytestmark = pytest.mark.gpu


def _volume(kind, dims):
    nx, ny, nz = dims
    if kind == "random":
        return synthetic.random_volume((nz, ny, nx), seed=nx)
    z, y, x = np.meshgrid(*(np.arange(n) + 0.5 for n in (nz, ny, nx)), indexing="ij")
    r = np.sqrt((x - nx / 2) ** 2 + (y - ny / 2) ** 2 + (z - nz / 2) ** 2)
    sd = r - 0.3 * min(dims)
    if kind == "shell":  # a band that never crosses zero: distances of one sign
        sd = np.abs(sd) + 0.4
    band = {"sphere": 3.0, "thin": 0.8, "shell": 2.0}[kind]
    t = np.trunc(np.clip(sd / band, -1, 1) * 32766).astype(np.int16)
    return np.stack([t, np.full(t.shape, 9, np.int16)], axis=-1)


@pytest.mark.parametrize("kind", ["random", "sphere", "thin", "shell"])
@pytest.mark.parametrize("dims,image", [((2, 2, 2), (9, 5)), ((33, 29, 41), (33, 17)), ((64, 16, 48), (8, 16)),
                                        ((71, 70, 69), (50, 31))])
def test_march(mcg, orc, kind, dims, image):
    vol = _volume(kind, dims)
    w, h = image
    gs = 0.02
    middle = np.array(dims) * gs / 2
    rng = np.random.default_rng(dims[0] + w)
    f = 0.8 * w
    K = (f, f, (w - 1) / 2.0, (h - 1) / 2.0)
    v = mcg.Voxel(torch.from_numpy(vol).cuda(), 0.05, 0.05, gs)
    for i in range(5):
        eye = middle + rng.uniform(-1, 1, 3) * np.array(dims) * gs * (0.9, 0.2, 0.5, 1.5, 0.0)[i]
        fwd = middle + rng.uniform(-0.1, 0.1, 3) * gs * min(dims) - eye
        fwd /= np.linalg.norm(fwd)
        right = np.cross([0.0, 1.0, 0.05], fwd)
        right /= np.linalg.norm(right)
        R = np.stack([right, np.cross(fwd, right), fwd], axis=1)
        d, n = mcg.raycast(v, mcg.intrinsic(*K), mcg.extrinsic(R, eye), w, h)
        ref = orc.raycast(vol, gs, orc.intrinsic(*K), orc.extrinsic(R, eye), w, h)
        assert np.array_equal(d.cpu().numpy().view(np.uint32), ref[0].view(np.uint32))
        assert np.array_equal(n.cpu().numpy().view(np.uint32), ref[1].view(np.uint32))
