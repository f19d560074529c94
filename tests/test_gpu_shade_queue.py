"""The warp's shading queue against the oracle: a faint TF under which a ray
leaves a hundred samples in it and one under which only a few rays leave any,
images whose last tiles are partly outside, every group size from one sample
to the whole warp, six and four taps, one view a launch and several.  The
sums are folded in sample order with the oracle's operations, so the images
are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 37, 21


@pytest.fixture(scope="module")
def scenes(rb, orc):
    vol = rb.phantom(128, seed=21)
    faint = rb.tf_build([(0, (20, 30, 40, 5)), (255, (220, 210, 200, 40))])
    sparse = rb.tf_build([(0, (0, 0, 0, 0)), (150, (90, 80, 70, 0)), (160, (250, 200, 150, 255)),
                          (255, (250, 250, 250, 255))])
    c = rb.Context(0)
    c.upload_volume(vol)
    c.shard_build(vol)
    c.bricks_build(vol, 1)
    page, pool = c.bricks_read()
    refs = {0: orc.CubeScene(vol), c.shard_mode: orc.ShardScene.build(vol),
            c.brick_mode: orc.BrickScene(page, pool)}
    yield c, refs, {"faint": faint, "sparse": sparse}
    c.close()


@pytest.mark.parametrize("group", [0, 1, 5, 31, 32])
@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("tf", ["faint", "sparse"])
def test_queue_equals_oracle(rb, orc, scenes, group, fast, tf):
    c, refs, tfs = scenes
    lut = tfs[tf]
    c.set_transfer(lut)
    c.set_quality(rb.QUALITY_FAST if fast else rb.QUALITY_FULL)
    try:
        for mode, ref in refs.items():
            views = []
            for i in range(2):
                p = rb.camera_view(0.7 + i, -0.5, 1.6, W, H, lut, step_voxels=0.5, frame_index=i)
                p.brick_mode = mode
                p.view_org = (i * W) | (i << 16)
                views.append(p)
            for persistent, vs in ((0, views[:1]), (0, views), (2, views)):
                c.set_schedule(persistent=persistent, shade_group=group)
                got = c.raycast(vs, 2 * W, H + 1)
                for v in vs:
                    want = orc.render(v, ref, lut, 2 * W, H + 1,
                                      quality=rb.QUALITY_FAST if fast else rb.QUALITY_FULL)[0]
                    x, y = v.view_org & 0xffff, v.view_org >> 16
                    assert np.array_equal(got[y:y + H, x:x + W], want[y:y + H, x:x + W])
    finally:
        c.set_quality(rb.QUALITY_FULL)
        c.set_schedule()
