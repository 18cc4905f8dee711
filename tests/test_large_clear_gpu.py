"""Frames with more pixels outside the volume's screen rectangle than are
cleared with the counters: their clear is a launch of its own, and every pixel
is written all the same, in both modes."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,rect", [(2560, 1440, None), (4096, 2048, (5, 3, 4000, 2000)), (1500, 1500, None)])
@pytest.mark.parametrize("sync", [True, False])
def test_large_frames_are_written_whole(gpu_ctx, W, H, rect, sync):
    import torch
    import livre_gb300 as lv
    vi = lv.VolumeInformation(64, 32, 1)
    vol = gpu_ctx.blob_volume(vi, 8, 3)
    tf = gpu_ctx.transfer_function(lv.linear_ramp_tf(64))
    mv, proj = lv.orbit_camera(1, 8, vi.world_size, W, H, radius_scale=5.0)
    outs = []
    for k, fill in enumerate((float("nan"), -7.0, 3.0)):
        out = torch.full((H, W, 4), fill, device="cuda")
        gpu_ctx.render(vol, tf, gpu_ctx.render_desc(mv, proj, W, H, sse=1.0, rect=rect, synchronous=sync or k == 0), out)
        outs.append(out)
    x, y, w, h = rect or (0, 0, W, H)
    assert gpu_ctx.last_stats()["n_samples"] > 0
    for out, fill in zip(outs[1:], (-7.0, 3.0)):
        assert torch.equal(out[y:y + h, x:x + w], outs[0][y:y + h, x:x + w])
        edge = out.clone()
        edge[y:y + h, x:x + w] = fill
        assert (edge == fill).all()
    assert torch.isfinite(outs[0][y:y + h, x:x + w]).all()
    vol.close()
    tf.close()
