"""An overlay atlas loaded from device memory that starts at any byte: the
atlas's texels bit for bit, and through an overlay view the quad words made
from them, against the same slots loaded from host memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1, 2, 3, 4])
def test_overlay_load_at_any_byte(rb, scroll_tf, off):
    import torch
    c = rb.Context(0)
    try:
        c.set_transfer(scroll_tf)
        c.bricks_build(rb.phantom((130, 90, 70), seed=3), 2)
        n = c.bricks_info()["nslots"] * 128 ** 3
        slots = np.random.default_rng(off).integers(0, 256, n, dtype=np.uint8)
        buf = torch.full((n + 64,), 255, dtype=torch.uint8, device="cuda")
        dev = buf[off:off + n]
        dev.copy_(torch.from_numpy(slots))
        torch.cuda.synchronize()
        p = rb.camera_view(0.7, -0.5, 1.6, 96, 72, scroll_tf, step_voxels=0.5)
        p.brick_mode = c.brick_mode
        p.overlay_flags, p.overlay_gain = 1 | (128 << 16), 1.5
        got = []
        for src in (slots, dev):
            c.overlay_load(0, src)
            assert np.array_equal(c.overlay_read(0).reshape(-1), slots)
            got.append(c.raycast(p, 96, 72))
        assert np.array_equal(got[0], got[1])
        assert got[0].any()
    finally:
        c.close()
