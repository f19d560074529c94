"""The adjoint's ray tiles and its common reverse loops at their edges:
views of one pixel, of less and a little more than an 8 x 4 tile and of
unequal sizes in one call; every ray over the tape's 64 entries, none, and
both kinds in a warp (a faint TF on rays of unequal length); each checkpoint
interval, both accumulations, with and without the tape.  The forward is bit
equal to the FP32 oracle and the voxel and density-scale gradients within
1e-4 (relative L2) of the FP64 one; in deterministic mode every interval, with
and without the tape, gives the same bits; and FP32 atomics differ from them by
the rounding of their sums (an entry or voxel takes some 10^4 addends in any
order, 100 * 2^-24 expected, three times that allowed)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (7, 3), (9, 5), (33, 17), (8, 4)]


@pytest.fixture(scope="module")
def scene(rb):
    import torch
    rng = np.random.default_rng(11)
    vol = rb.phantom((57, 49, 61), seed=6).astype(np.float32) / 255.0
    vol = np.clip(vol + rng.normal(0, 0.03, vol.shape), -0.1, 1.1).astype(np.float32)
    views = []
    for i, (w, h) in enumerate(SIZES):
        v = rb.camera_view(0.4 + 1.1 * i, -0.4 + 0.2 * i, 1.5, w, h, rb.scroll_ramp_tf(),
                           step_voxels=0.5, max_mip=0.0, frame_index=i)
        v.density = 0.8 + 0.1 * i
        views.append(v)
    return vol, torch.tensor(vol, device="cuda"), views


def _lut(rb, kind):
    if kind == "scroll":
        return rb.scroll_ramp_tf().astype(np.float32) / 255.0
    top = 40 if kind == "faint" else 12
    return rb.tf_build([(0, (20, 30, 40, 6)), (255, (220, 210, 200, top))]).astype(np.float32) / 255.0


def _rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("kind", ["scroll", "faint", "fainter"])
def test_tiles_and_reverse_loops(rb, orc, ctx, scene, kind):
    import torch
    vol, dvol, views = scene
    lut = _lut(rb, kind)
    dlut = torch.tensor(lut, device="cuda")
    ctx.set_alpha_cutoff(0.98)
    n = sum(w * h * 3 for w, h in SIZES)
    rgb = torch.zeros(n, device="cuda")
    g = np.random.default_rng(4).normal(0, 1, n).astype(np.float32)
    dg = torch.tensor(g, device="cuda")
    rd, rs, off = np.zeros(vol.shape), 0.0, 0
    ctx.diff_forward(dvol, dlut, views, rgb, stream=ctx.stream, tape=True)
    torch.cuda.synchronize()
    out = rgb.cpu().numpy()
    for v, (w, h) in zip(views, SIZES):
        part = slice(off, off + w * h * 3)
        want = np.asarray(orc.diff_forward32(v, vol, lut, 0.98)[0]).reshape(-1)
        assert np.array_equal(out[part], want)
        _, d, _, s = orc.diff_grad64(v, vol, lut, g[part].reshape(h, w, 3), 0.98, decisions32=True)
        rd, rs, off = rd + d, rs + s, off + w * h * 3
    exact = {}
    for k in (32, 64, 128):
        for det in (True, False):
            for tape in (False, True):
                gd, gl = torch.empty_like(dvol), torch.empty_like(dlut)
                gs = torch.empty(1, device="cuda")
                ctx.raycast_bwd(dvol, dlut, views, dg, gd, gl, gs, k, det, stream=ctx.stream, tape=tape)
                torch.cuda.synchronize()
                assert _rel(gd.cpu().numpy(), rd) < 1e-4
                assert abs(gs.item() - rs) <= 1e-4 * abs(rs)
                got = (gd.cpu(), gl.cpu(), gs.cpu())
                for a, b in zip(got, exact.setdefault("first", got)):
                    assert torch.equal(a, b) if det else _rel(a.numpy(), b.numpy()) < 2e-5
