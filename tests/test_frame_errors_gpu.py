"""After lv_render has returned an error, the frame belongs to the caller again
in stream order: what the caller writes on its stream stays, although the
frame's clear was queued on the library's own stream."""
import pytest

pytestmark = pytest.mark.gpu


# 2048 x 1024 pixels are cleared with the frame's counters, more in a launch of their own
@pytest.mark.parametrize("W,H", [(512, 512), (2048, 1024), (2560, 1440), (4096, 4096)])
@pytest.mark.parametrize("sync", [True, False])
def test_frame_is_the_callers_after_an_error(gpu_ctx, native, W, H, sync):
    import torch
    import livre_gb300 as lv
    vi = lv.VolumeInformation(64, 32, 1)
    vol = gpu_ctx.blob_volume(vi, 8, 3)
    tf = gpu_ctx.transfer_function(lv.linear_ramp_tf(64))
    mv, proj = lv.orbit_camera(1, 8, vi.world_size, W, H, radius_scale=6.0)
    desc = gpu_ctx.render_desc(mv, proj, W, H, sse=1.0, synchronous=sync)
    # a synchronous frame, after which every brick is resident
    good = gpu_ctx.render(vol, tf, gpu_ctx.render_desc(mv, proj, W, H, sse=1.0)).clone()
    for _ in range(4):
        out = torch.full((H, W, 4), 3.0, device="cuda")
        torch.cuda._sleep(2_000_000)  # the frame's clear waits for the caller's earlier work
        lv.check(native.lv_test_fail_frame(gpu_ctx.handle), gpu_ctx.handle)
        with pytest.raises(lv.LivreError):
            gpu_ctx.render(vol, tf, desc, out)
        # the last rows, which the clear reaches last
        out[-8:] = 5.0
        torch.cuda.synchronize()
        assert (out[-8:] == 5.0).all()
        # the next frame is whole
        gpu_ctx.render(vol, tf, desc, out)
        assert torch.equal(out, good) and gpu_ctx.last_stats()["error_flags"] == 0
    vol.close()
    tf.close()
