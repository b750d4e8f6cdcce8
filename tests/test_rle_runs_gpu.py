"""Runs against the encoder's and the decoder's splits: run lengths around 4
voxels (a 16-byte word), 128 (a warp's segment), 4096 (a chunk), 16383 (a
record), slices whose starts fall on every 4-byte offset, volumes at every
offset from a 16-byte boundary; both formats.  The host codec is the oracle
of both directions, byte for byte."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 4, 5, 7, 8, 127, 128, 129, 130, 255, 256, 4095, 4096, 4097, 8191, 16382, 16383, 16384, 16385, 32766, 32767, 40000]


def _volume(shape, seed, short):
    nz, ny, nx = shape
    rng = np.random.default_rng(seed)
    n = nx * ny * nz
    out = np.empty((n, 2), np.int16)
    at = 0
    while at < n:
        length = int(rng.choice(LENGTHS[:9] if short else LENGTHS))
        kind = rng.integers(0, 4)
        t = (32766, -32766, int(rng.integers(-32767, 32768)), int(rng.integers(-5, 6)))[kind]
        end = min(n, at + length)
        out[at:end, 0] = t
        # weights change inside runs now and then: records of the lossless format split there
        out[at:end, 1] = 0 if rng.random() < 0.5 else int(rng.integers(-32768, 32768))
        if rng.random() < 0.2:
            out[at:end, 1] = rng.integers(0, 3, end - at)
        at = end
    return out.reshape(nz, ny, nx, 2)


@pytest.mark.parametrize("lossless", [False, True])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 1, 5), (5, 7, 3), (4, 33, 64), (3, 63, 65), (2, 301, 143), (3, 256, 256)])
def test_both_ways(mcg, shape, offset, lossless):
    nz, ny, nx = shape
    n = nx * ny * nz
    for seed, short in ((1, False), (2, True)):
        vol = _volume(shape, seed, short)
        image = bytes(mcg.rle_encode_host(vol, 0.1, 0.2, 0.3, lossless))
        buf = torch.zeros((n + 8, 2), dtype=torch.int16, device="cuda")
        view = buf[offset:offset + n].view(nz, ny, nx, 2)
        view.copy_(torch.from_numpy(vol))
        got = bytes(mcg.rle_encode(mcg.Voxel(view, 0.1, 0.2, 0.3), lossless))
        assert got == image
        back = torch.full((n + 8, 2), 77, dtype=torch.int16, device="cuda")
        ctx = mcg.default_context()
        arr = np.frombuffer(image, np.uint8)
        st = mcg._lib.mcg_rle_decode(ctx.handle, arr.ctypes.data_as(ctypes.c_void_p), arr.size,
                                     ctypes.c_void_p(back.data_ptr() + 4 * offset), n,
                                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == 0
        torch.cuda.synchronize()
        want, _ = mcg.rle_decode_host(image)
        assert np.array_equal(back[offset:offset + n].cpu().numpy().reshape(vol.shape), want)
        assert bool((back[:offset] == 77).all()) and bool((back[offset + n:] == 77).all())


@pytest.mark.parametrize("offset", [0, 3])
@pytest.mark.parametrize("shape", [(2, 256, 256), (2, 257, 255), (3, 256, 257), (2, 300, 500), (3, 1, 200001), (1, 640, 1000)])
def test_long_chunks_in_parts(mcg, shape, offset):
    """Slices of one run, of runs that end around multiples of 65536 voxels
    (where a chunk's parts end), and of short runs then one long run."""
    nz, ny, nx = shape
    xy, n = nx * ny, nx * ny * nz
    rng = np.random.default_rng(nx + offset)
    for kind in range(3):
        vol = np.zeros((nz, xy, 2), np.int16)
        for z in range(nz):
            if kind == 0:
                vol[z] = (32766, -32766, 5)[z], 0
            elif kind == 1:
                cuts = [c for c in (3 * z, 65535 - z, 65536, 65537 + z, 131072, 131075) if c < xy]
                for a, b in zip([0] + cuts, cuts + [xy]):
                    vol[z, a:b, 0] = rng.integers(-1000, 1000)
            else:
                at = int(rng.integers(2000, min(xy, 9000)))
                vol[z, :at, 0] = rng.integers(-3, 3, at)
                vol[z, at:, 0] = -32766
                vol[z, xy - 5:, 0] = np.arange(5)
        vol = vol.reshape(nz, ny, nx, 2)
        image = bytes(mcg.rle_encode_host(vol, 0.1, 0.2, 0.3, False))
        back = torch.full((n + 8, 2), 77, dtype=torch.int16, device="cuda")
        ctx = mcg.default_context()
        arr = np.frombuffer(image, np.uint8)
        st = mcg._lib.mcg_rle_decode(ctx.handle, arr.ctypes.data_as(ctypes.c_void_p), arr.size,
                                     ctypes.c_void_p(back.data_ptr() + 4 * offset), n,
                                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == 0
        torch.cuda.synchronize()
        want, _ = mcg.rle_decode_host(image)
        assert np.array_equal(back[offset:offset + n].cpu().numpy().reshape(vol.shape), want)
        assert bool((back[:offset] == 77).all()) and bool((back[offset + n:] == 77).all())
