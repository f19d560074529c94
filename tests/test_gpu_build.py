"""The brick cache's device builders at the edges of their tiles: extents of
one brick, one voxel past a brick and odd rows (whose words are not
aligned), from host memory and from device memory at odd addresses, one
context rebuilt with caches of other sizes (its buffers are kept or
replaced).  Page table and slots bit for bit against the oracle's builder;
the quad words and block maxima through MIP and step-heatmap views, whose
bytes and step counts depend on each of them; overlay atlases bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (nx, ny, nz), levels, min_max, device offset in bytes (None: host array)
CASES = [((128, 128, 128), 1, 0, None), ((129, 257, 130), 2, 0, 3), ((301, 77, 200), 3, 60, 1),
         ((256, 256, 128), 2, 0, 16), ((260, 131, 129), 2, 30, 4), ((64, 40, 33), 1, 0, 2)]


@pytest.fixture(scope="module")
def one(rb, scroll_tf):
    c = rb.Context(0)
    c.set_transfer(scroll_tf)
    yield c
    c.close()


def _device(vol, off):
    import torch
    buf = torch.full((vol.size + 64,), 255, dtype=torch.uint8, device="cuda")
    view = buf[off:off + vol.size].view(vol.shape)
    view.copy_(torch.from_numpy(vol))
    torch.cuda.synchronize()
    return view


@pytest.mark.parametrize("case", range(len(CASES)))
def test_bricks_build_edges(rb, orc, one, scroll_tf, case):
    (nx, ny, nz), nlev, min_max, off = CASES[case]
    vol = rb.phantom((nx, ny, nz), seed=40 + case)
    vol[-3:, -2:, -5:] = 250  # the far corner counts
    one.bricks_build(vol if off is None else _device(vol, off), nlev, min_max)
    ref = orc.BrickScene.build(vol, nlev, min_max=min_max)
    page, pool = one.bricks_read()
    assert np.array_equal(page, ref.page)
    assert np.array_equal(pool, ref.pool)
    w, h = 96, 72
    m = float(max(nx, ny, nz))
    for mode in (rb.MODE_MIP, rb.MODE_HEATMAP, rb.MODE_FULL):
        p = rb.camera_view(0.9, -0.5, 1.7, w, h, scroll_tf, target=(nx / m / 2, ny / m / 2, nz / m / 2),
                           step_voxels=0.5, mode=mode)
        p.brick_mode = one.brick_mode
        steps = np.zeros((h, w), np.uint32)
        got = one.raycast(p, w, h, steps=steps)
        want, rsteps, _, _, _ = orc.render(p, ref, scroll_tf, w, h)
        assert np.array_equal(got, want)
        assert np.array_equal(steps, rsteps)
    for which in (1, 2):  # box pyramid and label strides
        o = rb.phantom((nx, ny, nz), seed=70 + case)
        one.overlay_build(which, o if off is None else _device(o, off))
        slots = np.asarray(ref.build_overlay(which, o)).reshape(-1)
        assert np.array_equal(one.overlay_read(which).reshape(-1), slots)


@pytest.mark.parametrize("edge", [128, 384])
def test_shard_maxima(rb, orc, one, edge):
    vol = rb.phantom(edge, seed=5)
    one.shard_build(vol)
    page, atlas = one.shard_read(0)
    b = edge // 128
    mx = vol.reshape(b, 128, b, 128, b, 128).max(axis=(1, 3, 5)).reshape(-1).astype(np.uint32)
    assert np.array_equal(page, np.arange(b ** 3, dtype=np.uint32) | (mx << 24))
    assert np.array_equal(atlas, vol)
