"""The section fills' row copies at odd sizes, bit for bit against the
oracle's tiles: rows that start at every alignment, are shorter than a word's
warp or end inside one, cells that reach past the volume on both axes, and
clipmap levels larger than the volume, over several window moves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,wz", [((5, 3, 9), 4), ((2047, 37, 9), 5), ((2101, 2049, 6), 4),
                                      ((33, 131, 12), 7)])
def test_slab_rows(rb, orc, shape, wz):
    nx, ny, nz = shape
    vol = np.random.default_rng(nx).integers(0, 256, (nz, ny, nx), dtype=np.uint8)
    c = rb.Context(0)
    try:
        c.slab_build(vol, wz, 0)
        for z0 in (0, 1, nz - wz):
            c.slab_window(z0)
            sc = orc.SlabScene(vol, wz, z0)
            for lev in range(sc.s.nlev):
                for k in range(sc.tiles[lev].shape[0]):
                    assert np.array_equal(c.slab_read(lev, k), sc.tiles[lev][k]), (z0, lev, k)
    finally:
        c.close()


@pytest.mark.parametrize("shape,depth", [((77, 53, 9), 3), ((2050, 61, 11), 5), ((4099, 2051, 7), 2)])
def test_clip_rows(rb, orc, shape, depth):
    nx, ny, nz = shape
    vol = np.random.default_rng(nx).integers(0, 256, (nz, ny, nx), dtype=np.uint8)
    c = rb.Context(0)
    try:
        c.clip_build(vol, depth)
        prev = None
        for fx, fy, z0 in ((0.6 * nx, 0.5 * ny, 0), (0.6 * nx, 0.5 * ny, 1), (0.1 * nx, 0.9 * ny, 2)):
            c.clip_frame(fx, fy, z0)
            prev = orc.clip_origins(nx, ny, fx, fy, prev)
            sc = orc.ClipScene(vol, depth, prev, z0)
            for l in range(6):
                for k in range(sc.tex[l].shape[0]):
                    assert np.array_equal(c.clip_read(l, k), sc.tex[l][k]), (z0, l, k)
    finally:
        c.close()


@pytest.mark.parametrize("shape,win", [((301, 277, 14), (301, 277, 5, 2)), ((1301, 877, 20), (640, 480, 7, 3))])
def test_vslab_rows(rb, orc, shape, win):
    nx, ny, nz = shape
    vol = np.random.default_rng(nx).integers(0, 256, (nz, ny, nx), dtype=np.uint8)
    c = rb.Context(0)
    try:
        c.vslab_begin(vol, *win)
        sc = orc.VSlabScene(vol, *win)
        for i in range(7):
            f = (0.5 * nx + 90 * i, 0.5 * ny - 40 * i, min(i, nz - win[2] - 1))
            st = c.vslab_frame(*f, 40)
            assert st["jobs"] == len(sc.frame(*f, 40))
            for k in range(sc.v["ntiles"]):
                assert np.array_equal(c.vslab_read(k), sc.tiles[k]), (i, k)
            assert np.array_equal(c.vslab_table(), np.asarray(sc.table).reshape(-1, 4))
    finally:
        c.close()
