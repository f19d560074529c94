"""Differentiable calls of one context that overlap on several streams over
one density: two forwards, a taped one beside a validation one, a forward
beside an atomic backward, forwards of other transfer functions, more calls
in flight than the context's ring has slots.  Renders and step totals are the
bits of the same calls in order; FP32 atomics differ by the rounding of their
sums (a voxel or entry takes some 10^4 addends in any order: 100 * 2^-24
relative expected, three times that allowed)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H, N = 150, 117, 10


@pytest.fixture(scope="module")
def scene(rb):
    import torch
    rng = np.random.default_rng(3)
    vol = rb.phantom((90, 83, 97), seed=8).astype(np.float32) / 255.0
    vol = torch.tensor(np.clip(vol + rng.normal(0, 0.03, vol.shape), 0, 1).astype(np.float32), device="cuda")
    luts = []
    for top in (12, 200):
        lut = rb.tf_build([(0, (20, 30, 40, 3)), (255, (220, 210, 200, top))])
        luts.append(torch.tensor(lut.astype(np.float32) / 255.0, device="cuda"))
    luts.append(torch.tensor(rb.scroll_ramp_tf().astype(np.float32) / 255.0, device="cuda"))
    sets = []
    for s in range(3):
        views = []
        for i in range(N):
            v = rb.camera_view(0.3 + 0.7 * i + 0.2 * s, -0.4 + 0.1 * s, 1.4, W - 7 * s, H + s, rb.scroll_ramp_tf(),
                               step_voxels=0.5, max_mip=0.0, frame_index=i)
            views.append(v)
        sets.append(views)
    c = rb.Context(0)
    yield c, vol, luts, sets
    c.close()


def _size(views):
    return sum(v.viewport[0] * v.viewport[1] * 3 for v in views)


class Forward:
    def __init__(self, scene, views, lut, tape=False):
        import torch
        self.ctx, self.vol = scene[0], scene[1]
        self.views, self.lut, self.tape = views, lut, tape
        self.rgb = torch.zeros(_size(views), device="cuda")
        self.total = torch.zeros(1, dtype=torch.int64, device="cuda")

    def clear(self):
        self.rgb.fill_(-1.0)
        self.total.zero_()

    def run(self, stream):
        self.ctx.diff_forward(self.vol, self.lut, self.views, self.rgb, total=self.total, stream=stream,
                              tape=self.tape)

    def result(self):
        return [self.rgb.clone(), self.total.clone()]

    def check(self, want):
        for a, b in zip(self.result(), want):
            assert (a == b).all()


class Backward:
    def __init__(self, scene, views, lut):
        import torch
        self.ctx, self.vol = scene[0], scene[1]
        self.views, self.lut = views, lut
        g = torch.Generator(device="cuda").manual_seed(2)
        self.grad = torch.randn(_size(views), device="cuda", generator=g)
        self.out = [torch.zeros_like(self.vol), torch.zeros_like(lut), torch.zeros(1, device="cuda")]

    def clear(self):
        for o in self.out:
            o.fill_(-1.0)

    def run(self, stream):
        self.ctx.raycast_bwd(self.vol, self.lut, self.views, self.grad, *self.out, 64, False, stream=stream)

    def result(self):
        return [o.clone() for o in self.out]

    def check(self, want):
        for a, b in zip(self.out, want):
            assert (a - b).double().norm() <= 300 * 2.0 ** -24 * b.double().norm()


def _overlap(calls, rounds=12):
    import torch
    want = []
    for c in calls:
        c.clear()
        torch.cuda.synchronize()
        c.run(0)
        torch.cuda.synchronize()
        want.append(c.result())
    streams = [torch.cuda.Stream() for _ in calls]
    for _ in range(rounds):
        for c in calls:
            c.clear()
        torch.cuda.synchronize()
        for c, s in zip(calls, streams):
            c.run(s.cuda_stream)
        torch.cuda.synchronize()
        for c, w in zip(calls, want):
            c.check(w)


def test_two_forwards(scene):
    _overlap([Forward(scene, scene[3][0], scene[2][0]), Forward(scene, scene[3][1], scene[2][0])])


def test_taped_beside_validation(scene):
    _overlap([Forward(scene, scene[3][0], scene[2][0], tape=True), Forward(scene, scene[3][2], scene[2][0])])


def test_forward_beside_backward(scene):
    _overlap([Forward(scene, scene[3][0], scene[2][0]), Backward(scene, scene[3][1], scene[2][0])])


def test_other_transfer_functions(scene):
    _overlap([Forward(scene, scene[3][0], scene[2][k]) for k in range(3)])


def test_more_calls_than_ring_slots(scene):
    _overlap([Forward(scene, scene[3][k % 3], scene[2][0]) for k in range(6)] +
             [Backward(scene, scene[3][1], scene[2][0])], rounds=4)
