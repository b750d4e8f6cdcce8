"""What the encoder needs beside the volume and the image: for slices far smaller
than its chunks of 4096 voxels a part of the volume, not 536 bytes a slice; and
more slices than are taken in hand at a time give the bytes of the slices
themselves.  Oracle: the host encoder."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _volume(shape, seed):
    rng = np.random.default_rng(seed)
    n = int(np.prod(shape))
    t = np.repeat(rng.choice(np.array([32766, -32766, 5, -7], np.int16), n), rng.integers(1, 40, n))[:n]
    w = np.where(rng.random(n) < 0.9, 1, 3).astype(np.int16)
    return np.stack([t, w], axis=-1).reshape(*shape, 2)


@pytest.mark.parametrize("xy", [(1, 1), (1, 3), (8, 8), (31, 1), (32, 1), (33, 1), (63, 65), (64, 64), (17, 241), (4100, 1)])
@pytest.mark.parametrize("lossless", [False, True])
def test_short_slices(mcg, xy, lossless):
    vol = _volume((50, xy[1], xy[0]), seed=xy[0])
    ctx = mcg.Context()
    for v in (vol, vol[:7], vol):  # on scratch of other sizes too
        t = mcg.Voxel(torch.from_numpy(np.ascontiguousarray(v)).cuda(), 0.03, 0.03, 0.01)
        assert mcg.rle_encode(t, lossless=lossless, ctx=ctx) == mcg.rle_encode_host(v, 0.03, 0.03, 0.01, lossless=lossless)


def test_scratch_of_short_slices(mcg):
    nz = 1000000
    vol = torch.zeros((nz, 8, 8, 2), dtype=torch.int16, device="cuda")
    vol[..., 0] = 32766
    v = mcg.Voxel(vol, 0.03, 0.03, 0.01)
    ctx = mcg.Context()
    # (what the runtime loads with a kernel's first launch is loaded here)
    image = mcg.rle_encode(mcg.Voxel(vol[:10].contiguous(), 0.03, 0.03, 0.01), ctx=ctx)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    whole = bytes(mcg.rle_encode(v, ctx=ctx))
    used = before - torch.cuda.mem_get_info()[0]
    assert len(image) == 40 + 10 * 6 and whole[40:] == bytes(image)[40:46] * nz
    # slices' sizes and offsets 16 MB, marks 8, chunk records 24, image 6, in steps of 2 MB
    assert used <= (16 + 8 + 24 + 6 + 16) << 20


def test_more_slices_than_in_hand(mcg):
    base = _volume((20, 1024, 1024), seed=5)
    nz = 2300  # 2200 slices of 1024 x 1024 are taken at a time
    big = torch.from_numpy(base).cuda()[torch.arange(nz, device="cuda") % 20]
    out = bytearray(mcg.rle_encode_host(base, 0.03, 0.03, 0.01, lossless=True))
    got = np.frombuffer(mcg.rle_encode(mcg.Voxel(big, 0.03, 0.03, 0.01), lossless=True), np.uint8)
    body = np.frombuffer(out, np.uint8)[40:]
    assert got.size == 40 + body.size * (nz // 20)
    assert bytes(got[:24]) == bytes(out[:24]) and int(got[24:28].view(np.int32)[0]) == nz
    assert np.array_equal(got[40:].reshape(nz // 20, -1), np.broadcast_to(body, (nz // 20, body.size)))
