"""Several frames integrated in one call inside a CUDA graph: taken together
where an earlier call has sized the scratch for that, frame by frame where it
has only been sized for one, and right again when replayed after calls that
outgrew the scratch of either.  Oracle: frame by frame, every byte."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DIMS, FRAMES = (40, 24, 32), 5


class Loop:
    def __init__(self, mcg, orc, image, vtype):
        self.mcg, self.orc = mcg, orc
        self.h, self.w = image
        self.trunc, self.gs = 0.08, 1.0 / 40
        args = (0.8 * max(image), 0.8 * max(image), (self.w - 1) / 2.0, (self.h - 1) / 2.0)
        self.k, self.ko = mcg.intrinsic(*args), orc.intrinsic(*args)
        self.v = mcg.voxel_new(DIMS, self.trunc, self.trunc, self.gs, dtype=vtype)
        self.ref = self.v.data.cpu().numpy().copy()
        self.poses = [(np.eye(3), np.array([0.5 + 0.02 * i, 0.3, -0.4])) for i in range(FRAMES)]
        self.pt = torch.stack([mcg.extrinsic_tensor(R, t) for R, t in self.poses]).contiguous()
        self.m = torch.zeros((FRAMES, self.h, self.w), device="cuda")  # no valid pixel
        self.rng = np.random.default_rng(self.w)

    def call(self, n=FRAMES):
        self.mcg._integrate_frames(self.v, self.k, self.pt[:n], self.m[:n], None, False)

    def capture(self, stream):
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph, stream=stream):
            self.call()

    def replay(self):
        d = self.rng.uniform(0.5, 1.2, (FRAMES, self.h, self.w)).astype(np.float32)
        self.m.copy_(torch.from_numpy(d))
        torch.cuda.synchronize()
        self.graph.replay()
        torch.cuda.synchronize()
        for f, (R, t) in enumerate(self.poses):
            self.orc.integrate(self.ref, self.trunc, self.trunc, self.gs, self.ko, self.orc.extrinsic(R, t), d[f], None)
        assert (self.ref[..., 1] != 0).any()
        assert np.array_equal(self.v.data.cpu().numpy(), self.ref)


@pytest.fixture
def fresh(mcg, monkeypatch):
    """the calls below on a context of their own, its scratch not yet sized"""
    ctx = mcg.Context()
    monkeypatch.setattr(mcg, "default_context", lambda device=None: ctx)
    yield ctx
    torch.cuda.synchronize()
    ctx.close()


@pytest.mark.parametrize("vtype", [torch.int16, torch.float32])
@pytest.mark.parametrize("warm", [FRAMES, 1])
def test_captured_frames(mcg, orc, fresh, warm, vtype):
    loop = Loop(mcg, orc, (30, 44), vtype)
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        loop.call(warm)
        st.synchronize()
        loop.capture(st)
    loop.replay()
    # a larger volume, larger images, more frames: every buffer of the scratch outgrown
    big = mcg.voxel_new((96, 80, 72), 0.03, 0.03, 1.0 / 96)
    n = 9
    mcg._integrate_frames(big, loop.k, loop.pt[:1].expand(n, 12).contiguous(),
                          torch.full((n, 160, 200), 0.8, device="cuda"), None, False)
    torch.cuda.synchronize()
    other = [torch.full((1 << 16,), 7, dtype=torch.int32, device="cuda") for _ in range(16)]
    loop.replay()
    loop.replay()
    assert all(bool((o == 7).all()) for o in other)


@pytest.mark.parametrize("warm,image", [((8, 64), (64, 8)), ((3, 300), (300, 3)), ((40, 40), (200, 8))])
@pytest.mark.parametrize("frames", [FRAMES, 1])
def test_capture_after_an_image_of_as_many_pixels(mcg, orc, fresh, warm, image, frames):
    """An earlier call of as many pixels sizes the scratch, whatever their layout."""
    loop = Loop(mcg, orc, image, torch.int16)
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        mcg._integrate_frames(loop.v, loop.k, loop.pt[:frames], torch.zeros((frames, *warm), device="cuda"), None, False)
        st.synchronize()
        loop.capture(st)
    loop.replay()
