"""Integrate's block list (blocks of 8^3 voxels that the frame can update)
at the sizes where it can go wrong: volumes with ragged blocks, images
with ragged depth tiles and images too small to hold a pixel, every option,
the pose on the host and on the device.  The oracle tests every voxel, so
the volumes have to be equal bit for bit."""
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
@pytest.mark.parametrize("dims,image", [((8, 8, 8), (64, 48)), ((9, 7, 17), (33, 25)), ((41, 30, 23), (47, 31)),
                                        ((36, 24, 40), (16, 8)), ((20, 20, 20), (2, 40)), ((20, 20, 20), (3, 3))])
def test_blocks_keep_every_update(mcg, orc, dims, image, vtype):
    rng = np.random.default_rng(sum(dims) + image[0])
    (nx, ny, nz), (w, h) = dims, image
    gs = 1.0 / max(dims)
    trunc = 2.5 * gs
    f = 0.9 * w
    k, ko = mcg.intrinsic(f, f, (w - 1) / 2.0, (h - 1) / 2.0), orc.intrinsic(f, f, (w - 1) / 2.0, (h - 1) / 2.0)
    v = mcg.voxel_new(dims, trunc, trunc, gs, dtype=vtype)
    ref = v.data.cpu().numpy().copy()
    middle = np.array(dims) * gs / 2
    for i in range(8):
        # outside, inside, and next to a face of the volume
        eye = middle + rng.uniform(-1, 1, 3) * (1.2, 0.3, 0.55)[i % 3]
        R = _look_at(eye, middle + rng.uniform(-0.2, 0.2, 3))
        m = rng.uniform(0.1, 1.6, (h, w)).astype(np.float32)
        m[rng.random((h, w)) < 0.3] = 0.0
        if i == 7:
            m[0, 0], m[h // 2, w // 2] = np.inf, np.nan
        n = rng.standard_normal((h, w, 3)).astype(np.float32)
        n[..., 2] = -np.abs(n[..., 2]) - 0.5
        n /= np.linalg.norm(n, axis=-1, keepdims=True)
        n = n if i % 2 else None
        nd = None if n is None else torch.from_numpy(n).cuda()
        if i % 4 < 2:
            mcg.volumetric_integration(v, k, mcg.extrinsic(R, eye), torch.from_numpy(m).cuda(), nd, is_dynamic=i > 3)
        else:
            mcg.volumetric_integration_device_pose(v, k, mcg.extrinsic_tensor(R, eye), torch.from_numpy(m).cuda(), nd,
                                                   is_dynamic=i > 3)
        orc.integrate(ref, trunc, trunc, gs, ko, orc.extrinsic(R, eye), m, n, is_dynamic=i > 3)
    got = v.data.cpu().numpy()
    # an infinite depth has weight 0 and gives an empty float voxel 0 / 0,
    # a NaN whose bits no arithmetic fixes; everything else is equal in bits
    none = np.isnan(ref) if vtype == torch.float32 else np.zeros(ref.shape, bool)
    assert np.array_equal(np.isnan(got) if vtype == torch.float32 else none, none)
    bits = np.uint32 if vtype == torch.float32 else np.uint16
    assert np.array_equal(got.view(bits)[~none], ref.view(bits)[~none])
    if w > 2:
        assert (ref[..., 1] != 0).any()


def test_captured_integrate_outlives_larger_calls(mcg, orc):
    """A graph captured around a small volume's integrate still works after
    calls for a larger volume and image have outgrown the context's scratch."""
    rng = np.random.default_rng(7)
    k, ko = mcg.intrinsic(40.0, 40.0, 23.5, 17.5), orc.intrinsic(40.0, 40.0, 23.5, 17.5)
    v = mcg.voxel_new((32, 32, 32), 0.08, 0.08, 1.0 / 32)
    R, t = np.eye(3), np.array([0.5, 0.5, -0.6])
    pose = mcg.extrinsic_tensor(R, t)
    m = torch.zeros((36, 48), device="cuda")
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        mcg.volumetric_integration_device_pose(v, k, pose, m, None)  # no valid pixel: sizes the scratch only
        st.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            mcg.volumetric_integration_device_pose(v, k, pose, m, None)
    big = mcg.voxel_new((96, 80, 72), 0.03, 0.03, 1.0 / 96)
    kb = mcg.intrinsic(200.0, 200.0, 99.5, 79.5)
    mcg.volumetric_integration(big, kb, mcg.extrinsic(R, t), torch.full((160, 200), 1.0, device="cuda"), None)
    torch.cuda.synchronize()
    other = [torch.full((1 << 16,), 7, dtype=torch.int32, device="cuda") for _ in range(16)]
    ref = v.data.cpu().numpy().copy()
    for _ in range(2):
        d = rng.uniform(0.7, 1.4, (36, 48)).astype(np.float32)
        m.copy_(torch.from_numpy(d))
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        orc.integrate(ref, 0.08, 0.08, 1.0 / 32, ko, orc.extrinsic(R, t), d, None)
    assert (ref[..., 1] != 0).any()
    assert np.array_equal(v.data.cpu().numpy(), ref)
    assert all(bool((o == 7).all()) for o in other)


@pytest.mark.parametrize("vtype", [torch.int16, torch.float32])
@pytest.mark.parametrize("frames,with_normals", [(1, False), (2, True), (9, False), (33, True), (66, False)])
@pytest.mark.parametrize("dims,image", [((9, 7, 17), (33, 25)), ((32, 24, 40), (48, 32))])
def test_several_frames_in_one_pass(mcg, orc, dims, image, frames, with_normals, vtype):
    """Up to 32 frames go through the volume in one pass: equal to the
    oracle's frame by frame, at either side of 32 and with a remainder of 1."""
    rng = np.random.default_rng(sum(dims) + frames)
    (w, h), gs = image, 1.0 / max(dims)
    trunc, f = 2.5 * gs, 0.9 * image[0]
    k, ko = mcg.intrinsic(f, f, (w - 1) / 2.0, (h - 1) / 2.0), orc.intrinsic(f, f, (w - 1) / 2.0, (h - 1) / 2.0)
    v = mcg.voxel_new(dims, trunc, trunc, gs, dtype=vtype)
    ref = v.data.cpu().numpy().copy()
    middle = np.array(dims) * gs / 2
    poses = []
    for i in range(frames):
        eye = middle + rng.uniform(-1, 1, 3) * (1.2, 0.3, 0.55)[i % 3]
        poses.append((_look_at(eye, middle + rng.uniform(-0.2, 0.2, 3)), eye))
    m = rng.uniform(0.1, 1.6, (frames, h, w)).astype(np.float32)
    m[rng.random(m.shape) < 0.3] = 0.0
    n = rng.standard_normal((frames, h, w, 3)).astype(np.float32)
    n[..., 2] = -np.abs(n[..., 2]) - 0.5
    n /= np.linalg.norm(n, axis=-1, keepdims=True)
    pt = torch.stack([mcg.extrinsic_tensor(R, t) for R, t in poses]).contiguous()
    dyn = frames % 2 == 0
    mcg._integrate_frames(v, k, pt, torch.from_numpy(m).cuda(), torch.from_numpy(n).cuda() if with_normals else None,
                          dyn)
    for i, (R, t) in enumerate(poses):
        orc.integrate(ref, trunc, trunc, gs, ko, orc.extrinsic(R, t), m[i], n[i] if with_normals else None,
                      is_dynamic=dyn)
    assert np.array_equal(v.data.cpu().numpy(), ref)
    assert (ref[..., 1] != 0).any()
