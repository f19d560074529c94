"""The brick march's per-sample LOD, step and cached brick against the oracle
where their shortcuts end: axis-aligned orthographic rays that graze the
volume's faces (coordinates of exactly 0 and of its extent, directions with
zeros of both signs), a camera inside, far away (the top level) and close
(steps set by the ray's span), LOD biases past both ends, and extents that
are no multiple of a brick.  Images, step counts and MIP indices equal: both
sides run the same operations."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 61, 47
VIEWS = ["+x", "-x", "+y", "-z", "inside", "far", "close", "bias-9", "bias+2", "bias+30"]


@pytest.fixture(scope="module", params=[((150, 131, 260), 3), ((129, 300, 127), 2), ((60, 50, 40), 1)])
def scene(request, rb, orc, scroll_tf):
    shape, nlev = request.param
    c = rb.Context(0)
    c.set_transfer(scroll_tf)
    c.bricks_build(rb.phantom(shape, seed=11), nlev=nlev)
    yield c, orc.BrickScene(*c.bricks_read()), shape
    c.close()


def _view(rb, lut, what, shape, c):
    p = rb.camera_view(0.7, -0.4, {"far": 40.0, "close": 0.9}.get(what, 1.8), W, H, lut, step_voxels=0.6)
    p.brick_mode = c.brick_mode
    if what.startswith("bias"):
        p.lod_bias = float(what[4:])
    if what == "inside":
        p.cam_origin[0], p.cam_origin[1], p.cam_origin[2] = 0.25, 0.2, 0.2
    if what[0] in "+-" and len(what) == 2:
        a, sign = "xyz".index(what[1]), 1.0 if what[0] == "+" else -1.0
        u, v = (a + 1) % 3, (a + 2) % 3
        ext = [s / max(shape) for s in shape]
        zero = -0.0 if sign < 0 else 0.0
        fwd, right, up, org = [zero] * 3, [0.0] * 3, [0.0] * 3, [0.0] * 3
        fwd[a] = sign
        # the outermost pixel centres lie on the volume's faces
        right[u], up[v] = 0.5 * ext[u] * W / (W - 1), 0.5 * ext[v] * H / (H - 1)
        org[a] = -0.5 if sign > 0 else 1.5
        org[u], org[v] = 0.5 * ext[u], 0.5 * ext[v]
        for i in range(3):
            p.cam_forward[i], p.cam_right[i], p.cam_up[i], p.cam_origin[i] = fwd[i], right[i], up[i], org[i]
        p.view_flags = rb.VIEW_ORTHO
    return p


@pytest.mark.parametrize("what", VIEWS)
@pytest.mark.parametrize("mode", [0, 1, 2, 3, 5])
def test_steps(rb, orc, scroll_tf, scene, what, mode):
    c, ref, shape = scene
    p = _view(rb, scroll_tf, what, shape, c)
    p.mode = mode
    want, wsteps, wmip, _, st = orc.render(p, ref, scroll_tf, W, H)
    assert st == 0
    for sched in ({"persistent": 0}, {"persistent": 2}):
        c.set_schedule(**sched)
        steps, mip = np.zeros((H, W), np.uint32), np.zeros((H, W), np.uint32)
        got = c.raycast(p, W, H, steps=steps, mip_index=mip)
        assert np.array_equal(steps, wsteps), sched
        assert np.array_equal(got, want), sched
        if mode == rb.MODE_MIP:
            assert np.array_equal(mip, wmip), sched
    c.set_schedule()
