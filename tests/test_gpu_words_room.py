"""Quad words of a large volume are left out where they would take the
device's last quarter: the volume's allocation is then that of its bytes, and
the views are the same; a kept buffer that has room for them keeps them."""
import pytest

from fake_cudart import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["cube", "shard"])
def test_words_leave_room(tmp_path, kind):
    run(tmp_path, f"""
    import torch
    kind = {kind!r}
    vol = c.phantom((640, 640, 640), seed=3)  # 262 MB, and 1.2 GB of words
    torch.cuda.synchronize()
    n = vol.numel()

    def build(x):
        shim.shim_largest()
        x.upload_volume(vol) if kind == "cube" else x.shard_build(vol)
        return shim.shim_largest(), look(x, x.shard_mode if kind == "shard" else None)

    size, want = build(c)
    assert size > 5 * n
    d = rb.Context(0)
    d.set_transfer(lut)
    shim.shim_free(n + 5 * n)  # enough for the volume, under a quarter of any B200
    size, got = build(d)
    assert n < size < 1.3 * n
    assert np.array_equal(got, want)
    size, got = build(c)  # in the buffer that has them
    assert size < n and np.array_equal(got, want)
    d.close()
    """)
