"""Every pixel of the rendered rect is written, with the volume filling part,
all or none of the frame, and no pixel outside the rect."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,rect", [(1, 1, None), (97, 61, None), (300, 40, (3, 5, 251, 30)), (64, 300, (9, 280, 8, 20)),
                                      (200, 150, (0, 0, 7, 7))])
@pytest.mark.parametrize("center", [(0.0, 0.0, 0.0), (0.8, -0.6, 0.0), (30.0, 0.0, 0.0)])
def test_every_pixel_of_the_rect_is_written(gpu_ctx, W, H, rect, center):
    import torch
    import livre_gb300 as lv
    vi = lv.VolumeInformation(64, 32, 1)
    vol = gpu_ctx.blob_volume(vi, 8, 3)
    tf = gpu_ctx.transfer_function(lv.linear_ramp_tf(64))
    eye = (0.4, 0.9, 2.6)
    proj = lv.perspective(40.0, W / H, 0.1, 50.0)
    mv = lv.look_at(eye, center)
    outs = []
    for fill in (float("nan"), -7.0):
        out = torch.full((H, W, 4), fill, device="cuda")
        gpu_ctx.render(vol, tf, gpu_ctx.render_desc(mv, proj, W, H, sse=1.0, rect=rect), out)
        outs.append(out)
    x, y, w, h = rect or (0, 0, W, H)
    inside = torch.zeros((H, W), dtype=torch.bool, device="cuda")
    inside[y:y + h, x:x + w] = True
    assert torch.isfinite(outs[0][inside]).all() and torch.equal(outs[0][inside], outs[1][inside])
    assert torch.isnan(outs[0][~inside]).all() and (outs[1][~inside] == -7.0).all()
    if center[0] > 10:
        assert (outs[1][inside] == 0).all() and gpu_ctx.last_stats()["n_samples"] == 0
    vol.close()
    tf.close()
