"""A volume rebuilt into its kept buffers beside other streams: while another
thread captures a stream (the rebuild is accepted and the capture stays
whole), and while a frame of the old volume still waits on a stream of the
caller's (the frame shows the old volume, the next one the new)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 64, 48


def _make(rb, kind, c, vol):
    if kind == "cube":
        c.upload_volume(vol)
    elif kind == "shard":
        c.shard_build(vol)
    else:
        c.bricks_postfilter(1 if kind == "filtered" else 0)
        c.bricks_build(vol, 2)


def _view(rb, kind, c, lut):
    p = rb.camera_view(0.6, -0.5, 1.8, W, H, lut, step_voxels=0.5)
    p.brick_mode = 0 if kind == "cube" else c.shard_mode if kind == "shard" else c.brick_mode
    return p


@pytest.mark.parametrize("kind", ["cube", "shard", "bricks", "filtered"])
def test_rebuild_while_another_thread_captures(rb, scroll_tf, kind):
    import torch
    vol = rb.phantom(128, seed=2)
    c = rb.Context(0)
    try:
        c.set_transfer(scroll_tf)
        _make(rb, kind, c, vol)
        want = c.raycast(_view(rb, kind, c, scroll_tf), W, H)
        x = torch.zeros(8, device="cuda")
        s = torch.cuda.Stream()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        failed = []

        def rebuild():
            try:
                _make(rb, kind, c, vol)
            except rb.R3DError as e:
                failed.append(e)

        with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
            x += 1
            t = threading.Thread(target=rebuild)
            t.start()
            t.join()
        assert not failed
        g.replay()
        torch.cuda.synchronize()
        assert x.tolist() == [1.0] * 8
        assert np.array_equal(c.raycast(_view(rb, kind, c, scroll_tf), W, H), want)
    finally:
        c.close()


@pytest.mark.parametrize("kind", ["cube", "shard", "bricks"])
def test_rebuild_behind_a_waiting_frame(rb, scroll_tf, kind):
    import torch
    vols = [rb.phantom(128, seed=k) for k in (2, 9)]
    c = rb.Context(0)
    try:
        c.set_transfer(scroll_tf)
        want = []
        for vol in vols:
            _make(rb, kind, c, vol)
            want.append(c.raycast(_view(rb, kind, c, scroll_tf), W, H))
        assert not np.array_equal(want[0], want[1])
        s = torch.cuda.Stream()
        out = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
        for k in (0, 1, 0):
            _make(rb, kind, c, vols[k])
            torch.cuda.synchronize()
            with torch.cuda.stream(s):
                torch.cuda._sleep(20_000_000)
            c.raycast(_view(rb, kind, c, scroll_tf), W, H, out=out, stream=s.cuda_stream)
            _make(rb, kind, c, vols[1 - k])
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), want[k])
            assert np.array_equal(c.raycast(_view(rb, kind, c, scroll_tf), W, H), want[1 - k])
    finally:
        c.close()
