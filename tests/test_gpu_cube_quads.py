"""The cube's and the shard atlas's quad words at odd extents, against the
oracle: volumes of one voxel, of extents below and past a word, of one texel
along an axis (whose mips clamp), from device memory at odd addresses, and a
context uploaded with other sizes in turn (its buffers are kept or replaced).
Mips and occupancy bit for bit; the words through views at every level (LOD
bias) in all modes, images and step counts equal; a batch planned over one
volume and launched over the next."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (3, 5, 2), (37, 1, 9), (64, 48, 33), (65, 31, 40), (130, 67, 71), (128, 64, 72)]
W, H = 45, 33


@pytest.fixture(scope="module")
def one(rb, scroll_tf):
    c = rb.Context(0)
    c.set_transfer(scroll_tf)
    yield c
    c.close()


@pytest.mark.parametrize("case", range(len(SHAPES)))
def test_cube(rb, orc, one, scroll_tf, case):
    import torch
    nx, ny, nz = SHAPES[case]
    vol = np.random.default_rng(case).integers(0, 256, (nz, ny, nx), dtype=np.uint8)
    buf = torch.zeros(vol.size + 8, dtype=torch.uint8, device="cuda")
    src = buf[case % 5:case % 5 + vol.size].view(vol.shape)
    src.copy_(torch.from_numpy(vol))
    torch.cuda.synchronize()
    one.upload_volume(src)
    ref = orc.CubeScene(vol)
    for m in range(-1, ref.c.nlevels):
        want = ref.occ if m < 0 else ref.levels[m]
        assert np.array_equal(one.cube_read(m), np.asarray(want).reshape(one.cube_read(m).shape)), m
    for mode in range(6):
        for bias, fast in ((0.0, False), (1.5, True)):
            one.set_quality(rb.QUALITY_FAST if fast else rb.QUALITY_FULL)
            p = rb.camera_view(0.8, -0.4, 1.9, W, H, scroll_tf, step_voxels=0.7, mode=mode,
                               lod_bias=bias, density=0.5)
            steps = np.zeros((H, W), np.uint32)
            got = one.raycast(p, W, H, steps=steps)
            img, rs, _, _, _ = orc.render(p, ref, scroll_tf, W, H, quality=int(fast))
            assert np.array_equal(got, img) and np.array_equal(steps, rs), (mode, bias)
    one.set_quality(rb.QUALITY_FULL)


def test_planned_batch_over_the_next_volume(rb, orc, scroll_tf):
    import torch
    c = rb.Context(0)
    try:
        c.set_transfer(scroll_tf)
        vols = [rb.phantom(n, seed=n) for n in (40, 72)]
        c.upload_volume(vols[0])
        views = [rb.camera_view(0.5 * i, -0.5, 2.0, W, H, scroll_tf, step_voxels=0.5, frame_index=i)
                 for i in range(3)]
        imgs = [torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda") for _ in views]
        b = rb.Batch(c, views, imgs)
        for vol in (vols[0], vols[1]):
            c.upload_volume(vol)
            for sched in ({"persistent": 0}, {"persistent": 1}, {"persistent": 2}):
                b.set_schedule(**sched)
                b.launch()
                torch.cuda.synchronize()
                for v, im in zip(views, imgs):
                    want = orc.render(v, orc.CubeScene(vol), scroll_tf, W, H)[0]
                    assert np.array_equal(im.cpu().numpy(), want)
        b.close()
    finally:
        c.close()
