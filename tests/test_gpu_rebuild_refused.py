"""A rebuild that is refused half way leaves the volume that was there, in a
kept buffer too: the copy of an upload, the display filter's scratch of a
shard build; and the next rebuild works."""
import pytest

from fake_cudart import run

pytestmark = pytest.mark.gpu


def test_cube_keeps_its_volume(tmp_path):
    run(tmp_path, """
    vols = [rb.phantom(96, seed=k) for k in (1, 2)]
    images = []
    for v in vols:
        c.upload_volume(v)
        images.append(look(c))
    assert not np.array_equal(*images)
    shim.shim_copy(1)
    refused(lambda: c.upload_volume(vols[0]), "InvalidValue")
    assert np.array_equal(look(c), images[1])
    assert np.array_equal(c.cube_read(0), vols[1])
    c.upload_volume(vols[0])
    assert np.array_equal(look(c), images[0])
    """)


def test_shard_keeps_its_atlas(tmp_path):
    run(tmp_path, """
    vols = [rb.phantom(128, seed=k) for k in (1, 2)]
    images = []
    for v in vols:
        c.shard_build(v)
        images.append(look(c, c.shard_mode))
    assert not np.array_equal(*images)
    c.bricks_postfilter(1)
    shim.shim_alloc(100 << 20, 1 << 40)  # the filter's scratch slots
    refused(lambda: c.shard_build(vols[0]), "NOMEM")
    assert np.array_equal(look(c, c.shard_mode), images[1])
    assert np.array_equal(c.shard_read(0)[1], vols[1])
    for n in range(1, 4):  # each of the copies of a build
        shim.shim_copy(n)
        c.bricks_postfilter(0)
        try:
            c.shard_build(vols[0])
        except rb.R3DError:
            assert shim.shim_refused() == 1
            assert np.array_equal(look(c, c.shard_mode), images[1])
    shim.shim_copy(0)
    shim.shim_alloc(1, 0)
    c.bricks_postfilter(0)
    c.shard_build(vols[0])
    assert np.array_equal(look(c, c.shard_mode), images[0])
    """)
