"""The ICP loop at image sizes around its work split (512 pixels a CTA): one
full CTA, one pixel row more, many CTAs with a ragged last one; one iteration
and the whole loop; a loop that fails.  The per-pixel arithmetic is the
oracle's bit for bit and the sums are binary64 in another order, so a pose
entry can round to a neighbouring binary32 per iteration: 4 iterations of at
most 2^-23 (entries below 2) stay below 1e-6."""
import math

import numpy as np
import pytest
import torch

import oracle
from icp_util import frames, pyramid_maps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bilinear", [False, True])
@pytest.mark.parametrize("size", [(31, 17), (32, 16), (40, 30), (97, 61), (160, 120)])
def test_loop_matches_oracle(mcg, size, bilinear):
    w, h = size
    d1, d2, _, (f, cx, cy) = frames(seed=1, w=w, h=h, f=0.75 * w)
    (v1, n1, k, _), = pyramid_maps(d1, f, cx, cy, levels=1)
    (v2, n2, _, _), = pyramid_maps(d2, f, cx, cy, levels=1)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    for it_max in (1, 12):
        ok, (r, t), iters, inl = oracle.icp(math.cos(math.radians(20)), 0.10, math.radians(20), 0.10, it_max, k,
                                            oracle.extrinsic(np.eye(3), np.zeros(3)), v1, n1, v2, n2, bilinear)
        got = torch.full((h, w), 7, dtype=torch.uint8, device="cuda")
        gok, pose, giters = mcg.icp(mcg.icp_params(it_max, bilinear), mcg.intrinsic(k.fx, k.fy, k.cx, k.cy),
                                    mcg.extrinsic(np.eye(3), np.zeros(3)), cu(v1), cu(n1), cu(v2), cu(n2), inlier=got)
        assert (gok, giters) == (ok, iters)
        if not ok:  # pose and inliers as they were
            assert list(pose.r) == [1, 0, 0, 0, 1, 0, 0, 0, 1] and list(pose.t) == [0, 0, 0]
            assert bool((got == 7).all())
            continue
        assert np.allclose(list(pose.r), r, rtol=0, atol=1e-6) and np.allclose(list(pose.t), t, rtol=0, atol=1e-6)
        if it_max == 1:  # the pass at the starting pose
            assert np.array_equal(got.cpu().numpy(), inl)
