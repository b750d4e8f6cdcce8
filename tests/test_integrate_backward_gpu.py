"""Integrate's adjoint where its work split changes: gradients on no voxel, on
one, on every voxel (full queues), on few of many; volumes smaller than one
scan; frames around a segment of 16; the gradients in two arrays and laid out
as the volume.  Oracle: the binary64 adjoint, relative 2-norm <= 1e-4 as for
the adjoint elsewhere; both layouts against each other within the order of
the atomics (1e-5)."""
import numpy as np
import pytest
import torch

from marching_cube_gb300 import synthetic

pytestmark = pytest.mark.gpu


def _rel(a, b):
    n = np.linalg.norm(b)
    return np.linalg.norm(a - b) / n if n else float(np.linalg.norm(a))


@pytest.mark.parametrize("frames,n", [(1, 6), (3, 40), (16, 24), (17, 24), (33, 17)])
@pytest.mark.parametrize("spread", ["all", "few", "one", "none"])
@pytest.mark.parametrize("dynamic", [False, True])
def test_gradient_patterns(mcg, orc, frames, n, spread, dynamic):
    scene = synthetic.BlendedSpheres(seed=1)
    w, h, f = 48, 36, 40.0
    depth, poses = scene.frames(frames, w=w, h=h, fx=f, fy=f)
    depth = depth.to(torch.float32)
    k, ko = mcg.intrinsic(f, f, (w - 1) / 2, (h - 1) / 2), orc.intrinsic(f, f, (w - 1) / 2, (h - 1) / 2)
    shape, gs = (n, n + 1, n - 1), 1.0 / n
    rng = np.random.default_rng(frames)
    g = rng.standard_normal(shape + (2,)).astype(np.float32)
    if spread == "few":
        g[rng.random(shape) > 0.03] = 0
    elif spread == "one":
        keep = g[n // 2, n // 2, n // 2].copy()
        g[:] = 0
        g[n // 2, n // 2, n // 2] = keep
    elif spread == "none":
        g[:] = 0
    trunc = 5 * gs
    pt = torch.stack([mcg.extrinsic_tensor(R, t) for R, t in poses])
    vol0 = np.stack([rng.uniform(-1, 1, shape), rng.uniform(0.5, 3, shape)], axis=-1).astype(np.float32)
    d, gd, v0 = depth.cuda(), torch.from_numpy(g).cuda(), torch.from_numpy(vol0).cuda()
    a = mcg.integrate_backward(shape, trunc, trunc, gs, k, pt, d, gd[..., 0], gd[..., 1], vol0=v0, is_dynamic=dynamic,
                               want_grad_vol0=True)
    b = mcg._integrate_backward(shape, trunc, trunc, gs, k, pt, d, None, None, v0, None, dynamic, None, True, None, None,
                                grad_vol=gd)
    want = orc.integrate_seq_backward_f64(shape, trunc, trunc, gs, ko, [orc.extrinsic(R, t) for R, t in poses],
                                          depth.numpy().astype(np.float64), g[..., 0].astype(np.float64),
                                          g[..., 1].astype(np.float64), vol0=vol0, is_dynamic=dynamic)
    for x, y, z in zip(a, b, want):
        x, y = x.cpu().numpy().astype(np.float64).reshape(-1), y.cpu().numpy().astype(np.float64).reshape(-1)
        z = np.asarray(z, np.float64).reshape(-1)
        assert _rel(x, z) <= 1e-4 and _rel(x, y) <= 1e-5
