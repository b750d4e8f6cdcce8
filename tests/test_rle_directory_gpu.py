"""A file's directory comes to the GPU piece by piece: while a piece expands, the
entries of later slices may still be those of another file decoded on the same
context.  300 equal slices of which 75 come after the first 64 MiB, after a
small file of as many slices, whose chunk numbers all lie below the large
file's; the volume itself is the expected result, and the host decoder's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _literals(nz, ny, nx, seed):
    """Every voxel differs from the one before: six bytes each, lossless."""
    rng = np.random.default_rng(seed)
    vol = np.empty((nz, ny, nx, 2), np.int16)
    vol[..., 0] = rng.integers(-30000, 30000, size=(nz, ny, nx))
    vol[..., 1] = (np.arange(nx * ny).reshape(ny, nx) % 2 + 1)[None]
    return vol


@pytest.mark.parametrize("before", [(3, 5), (40, 40)])
def test_file_after_a_smaller_one(mcg, tmp_path, before):
    nz = 300
    small, large = _literals(nz, *before, seed=1), _literals(nz, 100, 495, seed=2)
    ctx = mcg.Context()
    files = []
    for name, vol in (("small", small), ("large", large)):
        f = tmp_path / name
        f.write_bytes(mcg.rle_encode_host(vol, 0.03, 0.03, 0.01, lossless=True))
        files.append(str(f))
    per = 4 + 6 * 100 * 495
    assert ((64 << 20) - 40) // per == 225 and 40 + nz * per > (64 << 20)
    assert torch.equal(mcg.run_length_decode(files[0], ctx=ctx).data, torch.from_numpy(small).cuda())
    back = mcg.run_length_decode(files[1], ctx=ctx).data
    assert torch.equal(back, torch.from_numpy(large).cuda())
    assert np.array_equal(back.cpu().numpy(), mcg.rle_decode_host((tmp_path / "large").read_bytes())[0])
