"""Integrate's adjoint on either side of the volume size from which a CTA looks
at four voxels a thread at a time: gradients on every voxel (full queues), on
few, on one row in eight (some warps full, others empty), frames around one and
two segments of 16.  Oracle: the binary64 adjoint, relative 2-norm <= 1e-4 as
for the adjoint elsewhere."""
import numpy as np
import pytest
import torch

from marching_cube_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(85, 85, 85), (86, 85, 86)])  # x, y, z; 152 SMs: 622592 voxels
@pytest.mark.parametrize("frames,spread", [(3, "all"), (17, "few"), (17, "rows"), (33, "few")])
def test_rounds(mcg, orc, dims, frames, spread):
    nx, ny, nz = dims
    w, h, f = 40, 30, 34.0
    depth, poses = synthetic.BlendedSpheres(seed=2).frames(frames, w=w, h=h, fx=f, fy=f)
    depth = depth.to(torch.float32)
    k, ko = mcg.intrinsic(f, f, (w - 1) / 2, (h - 1) / 2), orc.intrinsic(f, f, (w - 1) / 2, (h - 1) / 2)
    shape, gs = (nz, ny, nx), 1.0 / nx
    trunc = 5 * gs
    rng = np.random.default_rng(frames)
    g = rng.standard_normal(shape).astype(np.float32)
    if spread == "few":
        g[rng.random(shape) > 0.02] = 0
    elif spread == "rows":
        g[:, np.arange(ny) % 8 != 3] = 0
    pt = torch.stack([mcg.extrinsic_tensor(R, t) for R, t in poses])
    got = mcg.integrate_backward(shape, trunc, trunc, gs, k, pt, depth.cuda(), torch.from_numpy(g).cuda(),
                                 want_grad_vol0=True)
    want = orc.integrate_seq_backward_f64(shape, trunc, trunc, gs, ko, [orc.extrinsic(R, t) for R, t in poses],
                                          depth.numpy().astype(np.float64), g.astype(np.float64),
                                          np.zeros(shape, np.float64))
    for x, z in zip(got, want):
        z = np.asarray(z, np.float64).reshape(-1)
        n = np.linalg.norm(z)
        d = np.linalg.norm(x.cpu().numpy().astype(np.float64).reshape(-1) - z)
        assert d <= 1e-4 * n if n else d == 0
