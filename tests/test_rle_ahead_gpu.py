"""Encoding on both sides of the size up to which the records are written before
the image's size has been read (8 MB at 6 bytes a voxel): the host encoder's bytes,
also after a call whose buffer was too small and after a larger volume's, and the
size asked for alone."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _volume(dims, seed):
    rng = np.random.default_rng(seed)
    n = int(np.prod(dims))
    t = np.repeat(rng.integers(-32766, 32767, n).astype(np.int16), rng.integers(1, 4, n))[:n]
    return np.stack([t, rng.integers(0, 3, n).astype(np.int16)], axis=-1).reshape(dims[2], dims[1], dims[0], 2)


@pytest.mark.parametrize("lossless", [False, True])
def test_small_volumes(mcg, lossless):
    ctx = mcg.Context()
    # 111^3 voxels are 8.2 MB, 111 x 113 x 112 8.4
    for i, dims in enumerate([(32, 32, 32), (111, 111, 111), (1, 1, 1), (111, 113, 112), (5, 7, 3), (64, 65, 63)]):
        vol = _volume(dims, i)
        want = bytes(mcg.rle_encode_host(vol, 0.05, 0.04, 0.01, lossless=lossless))
        t = torch.from_numpy(vol).cuda()
        size = ctypes.c_int64(-1)
        args = (ctx.handle, ctypes.c_void_p(t.data_ptr()), *dims, 0.05, 0.04, 0.01, 1 if lossless else 0)
        s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        small = np.full(len(want) - 1, 7, np.uint8)
        st = mcg._lib.mcg_rle_encode(*args, small.ctypes.data_as(ctypes.c_void_p), small.size, ctypes.byref(size), s)
        assert st == mcg.MCG_ERR_CAPACITY and size.value == len(want) and (small == 7).all()
        assert mcg._lib.mcg_rle_encode(*args, None, 0, ctypes.byref(size), s) == 0 and size.value == len(want)
        assert bytes(mcg.rle_encode(mcg.Voxel(t, 0.05, 0.04, 0.01), lossless=lossless, ctx=ctx)) == want
