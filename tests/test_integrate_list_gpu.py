"""Integrate on both sides of the number of blocks (8^3 voxels) from which the
blocks that a frame can update are listed: ragged blocks, thin volumes, images of
few and many depth tiles (blocks that cover one tile, a window of several rows
and more than are searched), the camera outside, inside and far away.  The oracle
tests every voxel, so the volumes have to be equal bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _look_at(eye, at):
    f = (at - eye) / np.linalg.norm(at - eye)
    r = np.cross([0.0, 1.0, 0.1], f)
    r /= np.linalg.norm(r)
    return np.stack([r, np.cross(f, r), f], axis=1)


@pytest.mark.parametrize("vtype", [torch.int16, torch.float32])
@pytest.mark.parametrize("dims", [(128, 128, 128), (129, 128, 128), (137, 129, 121), (7, 9, 40000)])
@pytest.mark.parametrize("image", [(31, 17), (130, 97), (640, 480)])
def test_both_sides(mcg, orc, dims, image, vtype):
    rng = np.random.default_rng(sum(dims) + image[0])
    w, h = image
    gs = 1.0 / min(max(dims), 128)
    trunc = 2.5 * gs
    f = 0.9 * w
    k, ko = mcg.intrinsic(f, f, (w - 1) / 2.0, (h - 1) / 2.0), orc.intrinsic(f, f, (w - 1) / 2.0, (h - 1) / 2.0)
    v = mcg.voxel_new(dims, trunc, trunc, gs, dtype=vtype)
    ref = v.data.cpu().numpy().copy()
    middle = np.minimum(np.array(dims) * gs / 2, 1.0)
    for i in range(4):
        eye = middle + rng.uniform(-1, 1, 3) * (1.2, 0.2, 0.55, 3.0)[i]
        R = _look_at(eye, middle + rng.uniform(-0.2, 0.2, 3))
        x, y = np.meshgrid(np.arange(w), np.arange(h))
        m = (np.linalg.norm(eye - middle) + 0.2 * np.sin(9.0 * x / w + i) * np.cos(7.0 * y / h)).astype(np.float32)
        m[rng.random((h, w)) < 0.05] = 0.0
        m[: h // 3, : w // 4] = 0.0  # tiles without a valid pixel
        mcg.volumetric_integration(v, k, mcg.extrinsic(R, eye), torch.from_numpy(m).cuda())
        orc.integrate(ref, trunc, trunc, gs, ko, orc.extrinsic(R, eye), m)
    bits = np.uint32 if vtype == torch.float32 else np.uint16
    assert np.array_equal(v.data.cpu().numpy().view(bits), ref.view(bits))
    assert (ref[..., 1] != 0).any()
