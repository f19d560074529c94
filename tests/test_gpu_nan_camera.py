"""Positions that are not numbers (a camera origin of NaN; an oblique slab
still gives its rays an interval to march) sample the brick cache at 0, as the
clamp of the oracle does, in the walked brick and in the cached one: images
and step counts bit for bit in every mode, over a cache of one brick and over
several levels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,nlev", [((60, 50, 40), 1), ((300, 140, 130), 2)])
def test_nan_origin(rb, orc, scroll_tf, shape, nlev):
    nx, ny, nz = shape
    vol = np.random.default_rng(5).integers(60, 90, (nz, ny, nx), dtype=np.uint8)
    vol[:4, :4, :4] = 150
    vol[-4:, -4:, -4:] = 240
    c = rb.Context(0)
    try:
        c.set_transfer(scroll_tf)
        c.bricks_build(vol, nlev)
        ref = orc.BrickScene.build(vol, nlev)
        w, h = 24, 16
        for mode in range(6):
            for axis in range(3):
                p = rb.camera_view(0.9, -0.5, 1.7, w, h, scroll_tf, step_voxels=0.5, mode=mode, density=0.05)
                p.brick_mode = c.brick_mode
                p.view_flags |= rb.VIEW_OBLIQUE
                p.slab_z0, p.slab_depth = 0.0, 24
                p.cam_origin[axis] = float("nan")
                steps = np.zeros((h, w), np.uint32)
                got = c.raycast(p, w, h, steps=steps)
                want, rsteps, _, _, _ = orc.render(p, ref, scroll_tf, w, h)
                assert steps.max() > 1 or mode == rb.MODE_RAYDIR  # (which does not march)
                assert np.array_equal(got, want), (mode, axis)
                assert np.array_equal(steps, rsteps), (mode, axis)
    finally:
        c.close()
