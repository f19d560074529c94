"""Cube and shard views of volumes whose quad words did not fit the memory
(a shim refuses their allocations): the kernels that sample bytes give the
images, step counts and projected indices of those that read words, in every
mode and schedule, and the oracle's images within 1/255; a batch over a scene
with words and one without draws both."""
import pytest

from fake_cudart import run

pytestmark = pytest.mark.gpu

BODY = """
import torch
import oracle as orc

def make(build, n, words):
    x = rb.Context(0)
    x.set_transfer(lut)
    if not words:  # room for the bytes alone, or a copy of them
        shim.shim_alloc(2 * n, 1 << 40)
    build(x)
    assert bool(shim.shim_refused()) != words
    shim.shim_alloc(1, 0)
    return x

def view(mode, mode_of, bias=0.0, frame=0):
    p = rb.camera_view(0.8, -0.4, 1.9, W, H, lut, step_voxels=0.7, mode=mode, lod_bias=bias,
                       density=0.5, frame_index=frame)
    p.brick_mode = mode_of
    return p

def draw(x, p, fast, persistent):
    steps, mip = np.zeros((H, W), np.uint32), np.zeros((H, W), np.uint32)
    x.set_quality(rb.QUALITY_FAST if fast else rb.QUALITY_FULL)
    x.set_schedule(persistent=persistent)
    n0 = shim.shim_launches()
    img = x.raycast(p, W, H, steps=steps, mip_index=mip)
    return {shim.shim_kernel(k) for k in range(n0, shim.shim_launches())}, img, steps, mip

def check(build, n, scene, mode_of):
    a, b = make(build, n, True), make(build, n, False)
    for mode in range(6):
        for bias, fast in ((0.0, 0), (1.5, 1)):
            p = view(mode, mode_of(a), bias)
            ref = orc.render(p, scene, lut, W, H, quality=fast)[0]
            for persistent in (0, 1, 2):
                ka, *wa = draw(a, p, fast, persistent)
                kb, *wb = draw(b, p, fast, persistent)
                assert ka != kb, "the same kernels"
                for u, v in zip(wa, wb):
                    assert np.array_equal(u, v), (mode, fast, persistent)
                assert np.abs(wb[0].astype(int) - ref.astype(int)).max() <= 1, (mode, fast)
    a.set_quality(rb.QUALITY_FULL)
    b.set_quality(rb.QUALITY_FULL)
    views = [view(rb.MODE_FULL, mode_of(a), 0.0, i) for i in range(4)]
    want = [draw(a, p, 0, 0)[1] for p in views]
    imgs = [torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda") for _ in views]
    plan = rb.Batch(a, views, imgs, scenes=[None, b, None, b])
    for persistent in (0, 2):
        plan.set_schedule(persistent=persistent)
        for im in imgs:
            im.zero_()
        torch.cuda.synchronize()
        plan.launch()
        torch.cuda.synchronize()
        for im, w in zip(imgs, want):
            assert np.array_equal(im.cpu().numpy(), w), persistent
    plan.close()
"""


@pytest.mark.parametrize("shape", [(65, 31, 40), (513, 1, 90), (128, 64, 72)])
def test_cube(tmp_path, shape):
    run(tmp_path, BODY + f"""
nx, ny, nz = {shape!r}
vol = np.random.default_rng(1).integers(0, 256, (nz, ny, nx), dtype=np.uint8)
check(lambda x: x.upload_volume(vol), vol.size, orc.CubeScene(vol), lambda x: 0)
""")


@pytest.mark.parametrize("slots", ["None", "np.array([5, 0xFFFFFFFF, 2, 7, 0, 0xFFFFFFFF, 1, 3], np.uint32)"],
                         ids=["identity", "shuffled"])
def test_shard(tmp_path, slots):
    run(tmp_path, BODY + f"""
slots = {slots}
vol = rb.phantom(256, seed=77)
check(lambda x: x.shard_build(vol, 2, slots), vol.size, orc.ShardScene.build(vol, 2, slots),
      lambda x: x.shard_mode)
""")


@pytest.mark.parametrize("kind", ["cube", "shard"])
def test_words_alone(tmp_path, kind):
    """Where words do not fit in one allocation with the bytes they are
    allocated alone, and go when the volume is replaced."""
    run(tmp_path, BODY + f"""
kind = {kind!r}
vols = [rb.phantom(128, seed=k) for k in (1, 2, 3)]

def build(x, k):
    x.upload_volume(vols[k]) if kind == "cube" else x.shard_build(vols[k])
    return x.shard_mode if kind == "shard" else 0

d = rb.Context(0)
d.set_transfer(lut)
want = []
shim.shim_largest()
for k in range(3):
    p = view(rb.MODE_FULL, build(c, k))
    want.append(draw(c, p, 0, 0)[:2])
    if k == 0:
        size = shim.shim_largest()
for k, whole in enumerate((False, False, True)):
    if not whole:
        shim.shim_alloc(size, size)
    build(d, k)
    assert bool(shim.shim_refused()) != whole
    shim.shim_alloc(1, 0)
    got = draw(d, p, 0, 0)[:2]
    assert got[0] == want[k][0], "another kernel"
    assert np.array_equal(got[1], want[k][1])
d.close()
""")
