"""n_launches of a frame is what was launched for it."""
import pytest

pytestmark = pytest.mark.gpu

# selection (an octree that fits one block), clear, residency pass, ray cast,
# counters to the host
SMALL = 5


def frames(ctx, lv, vol, tf, vi, W, H, radius=1.0, n=3, **kw):
    """n_launches of the last of n frames, and by how much the totals grew with it."""
    import torch
    mv, proj = lv.orbit_camera(1, 8, vi.world_size, W, H, radius_scale=radius)
    desc = ctx.render_desc(mv, proj, W, H, sse=1.0, **kw)
    for _ in range(n):
        before = ctx.totals()["launches"]
        ctx.render(vol, tf, desc)
        torch.cuda.synchronize()
    st = ctx.last_stats()
    assert st["error_flags"] == 0 and ctx.totals()["launches"] - before == st["n_launches"]
    return st["n_launches"]


def test_launches_of_resident_frames(gpu_ctx):
    import livre_gb300 as lv
    vi = lv.VolumeInformation(128, 32, 1)
    vol = gpu_ctx.blob_volume(vi, 8, 3)
    tf = gpu_ctx.transfer_function(lv.linear_ramp_tf(64))
    go = lambda *a, **kw: frames(gpu_ctx, lv, vol, tf, vi, *a, **kw)
    assert go(64, 48) == SMALL
    # the asynchronous residency pass counts the entries it kept in a launch of its own
    assert go(64, 48, synchronous=False) == SMALL + 1
    # more tiles than fit the GPU at once: their keys and their order
    assert go(1920, 1080) == SMALL + 2
    # more pixels to clear than go with the counters: a clear of their own
    assert go(4096, 2160, radius=3.0) == SMALL + 2 + 1
    vol.close()
    tf.close()


def test_launches_of_a_streaming_frame(gpu_ctx):
    import livre_gb300 as lv
    vi = lv.VolumeInformation(128, 32, 1)
    tf = gpu_ctx.transfer_function(lv.linear_ramp_tf(64))
    # bricks generated on the device (one launch) or gathered from the host store (one),
    # then the page table's update, the residency pass and the ray cast again
    for placement in (lv.BLOB_DEVICE, lv.BLOB_HOST):
        vol = gpu_ctx.blob_volume(vi, 8, 3, placement=placement)
        assert frames(gpu_ctx, lv, vol, tf, vi, 64, 48, n=1) == SMALL + 2 + 2
        vol.close()
    tf.close()
