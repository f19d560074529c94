"""The grid of a lane-refill launch is sized by the kernel it launches: the
occupancy that is asked for is that of the cube's and the atlas's kernels over
quad words when the views run those, and that of the view's own mode, in
direct, planned and allocation-free calls."""
import pytest

from fake_cudart import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["cube", "shard", "bricks"])
def test_grid_is_the_launched_kernels(tmp_path, kind):
    run(tmp_path, f"""
    import torch
    kind = {kind!r}
    vol = rb.phantom(128, seed=1)
    W, H = 1024, 768
    if kind == "cube":
        c.upload_volume(vol)
    elif kind == "shard":
        c.shard_build(vol)
    else:
        c.bricks_build(vol, 1)
    out = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = (W // 8 + 7) // 8 * ((H // 4 + 7) // 8) * 64
    c.set_schedule(persistent=1)
    for mode in (rb.MODE_FULL, rb.MODE_MIP, rb.MODE_FLAT):
        p = rb.camera_view(0.6, -0.5, 1.8, W, H, lut, step_voxels=0.5, mode=mode)
        p.brick_mode = dict(cube=0, shard=c.shard_mode, bricks=c.brick_mode)[kind]
        b = rb.Batch(c, [p], [out])
        b.set_schedule(persistent=1)
        calls = [lambda: c.raycast(p, W, H, out=out), lambda: b.launch(),
                 lambda: c._check(rb.lib.r3d_cuda_raycast_fwd_noalloc(
                     c.h, (rb.FrameParams * 1)(p), 1, out.data_ptr(), W, H, None))]
        for call in calls:
            n0 = shim.shim_launches()
            call()
            n1 = shim.shim_launches()
            blocks = ctypes.c_int()
            asked = shim.shim_asked(ctypes.byref(blocks))
            ours = [k for k in range(n0, n1) if shim.shim_kernel(k) == asked]
            assert ours, "the launched kernel is another one"
            assert shim.shim_grid(ours[-1]) == min(blocks.value * sms, (tiles + 3) // 4)
        torch.cuda.synchronize()
        b.close()
    """)
