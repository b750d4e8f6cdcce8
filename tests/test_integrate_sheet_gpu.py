"""Integrate into a sheet of more than 2^28 blocks of 8^3 voxels (69 GB): the
voxels of its first corner as in a small volume, those of its last corner found,
no others."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_sheet(mcg):
    ny, nz, gs = 131080, 131072, 1.0 / 64
    if torch.cuda.mem_get_info()[0] < 90 << 30:
        pytest.skip("90 GB of device memory")
    k = mcg.intrinsic(60.0, 60.0, 31.5, 23.5)
    R = np.array([[0.0, 0.0, 1.0], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0]])  # looks along x: image x along y, image y along z
    depth = torch.full((48, 64), 0.5, device="cuda")
    frames = [mcg.extrinsic(R, np.array([-0.49, y, z])) for y, z in ((1.0, 1.1), ((ny - 60) * gs, (nz - 50) * gs))]
    v = mcg.voxel_new((1, ny, nz), 5 * gs, 5 * gs, gs)
    small = mcg.voxel_new((1, 256, 256), 5 * gs, 5 * gs, gs)
    mcg.volumetric_integration(small, k, frames[0], depth)
    near = int((small.data[..., 1] != 0).sum())
    assert near > 500
    mcg.volumetric_integration(v, k, frames[0], depth)
    assert torch.equal(v.data[:256, :256], small.data)

    def updated():
        return sum(int((v.data[z:z + 8192, ..., 1] != 0).sum()) for z in range(0, nz, 8192))

    assert updated() == near
    mcg.volumetric_integration(v, k, frames[1], depth)
    far = int((v.data[-256:, -256:, ..., 1] != 0).sum())
    assert far > 500 and updated() == near + far
    del v
    torch.cuda.empty_cache()
