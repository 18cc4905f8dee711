"""Frames of few rays under the default launch (4 or 8 lanes share a ray):
image and sample count equal, bit for bit, those of the one-thread-per-pixel
launch, at viewports around its tiles and its ray-count thresholds, for both
filters, with and without overlap, for every kernel family."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# voxels, block, overlap, dtype (lv_dtype), filter
SPECS = [(96, 32, 1, 1, 1), ((128, 70, 64), 64, 1, 1, 1), (256, 128, 1, 1, 1), (60, 20, 2, 1, 1), (64, 16, 0, 1, 1),
         (64, 16, 0, 1, 0), (96, 32, 1, 2, 1), (130, 64, 1, 2, 1), (256, 128, 1, 2, 1), (72, 24, 1, 2, 1),
         (64, 16, 0, 2, 0)]
# about 0.8 of these pixels are candidate rays: from one tile to past 8192,
# 16384 and 81920
VIEWPORTS = [(1, 1), (3, 2), (5, 7), (33, 17), (97, 81), (121, 117), (147, 143), (331, 301)]


def both(ctx, lv, vol, tf, desc):
    import torch
    default = ctx.render_launch()
    img = ctx.render(vol, tf, desc)
    n = ctx.last_stats()
    try:
        ctx.set_render_launch(lv.LAUNCH_GRID, 8, 16)
        ref = ctx.render(vol, tf, desc)
        m = ctx.last_stats()
    finally:
        ctx.set_render_launch(**default)
    assert torch.equal(img, ref)
    assert n["n_samples"] == m["n_samples"] and n["error_flags"] == 0
    return img, n["n_samples"]


@pytest.mark.parametrize("voxels,block,overlap,dtype,filt", SPECS)
def test_split_frames_bit_identical(gpu_ctx, voxels, block, overlap, dtype, filt):
    import livre_gb300 as lv
    vi = lv.VolumeInformation(voxels, block, overlap, dtype=dtype)
    vol = gpu_ctx.blob_volume(vi, 12, 5, 3)
    tf = gpu_ctx.transfer_function(lv.gaussian_peaks_tf(128, seed=6))
    taken = 0
    for k, (W, H) in enumerate(VIEWPORTS):
        mv, proj = lv.orbit_camera(k, 8, vi.world_size, W, H, radius_scale=0.9)
        for early in (0.6, 2.0):
            desc = gpu_ctx.render_desc(mv, proj, W, H, sse=1.0, filt=filt, early_exit=early)
            taken += both(gpu_ctx, lv, vol, tf, desc)[1]
    assert taken > 10000
    vol.close()
    tf.close()


def test_split_rects_and_clip_planes(gpu_ctx):
    import livre_gb300 as lv
    vi = lv.VolumeInformation(96, 32, 1)
    vol = gpu_ctx.blob_volume(vi, 12, 5, 3)
    tf = gpu_ctx.transfer_function(lv.gaussian_peaks_tf(128, seed=6))
    mv, proj = lv.orbit_camera(1, 8, vi.world_size, 90, 70, radius_scale=0.8)
    planes = [(0.6, 0.0, 0.8, 0.1), (-1.0, 0.0, 0.0, 0.3)]
    for rect in (None, (7, 3, 33, 21), (40, 30, 1, 1)):
        desc = gpu_ctx.render_desc(mv, proj, 90, 70, sse=1.0, rect=rect, clip_planes=planes)
        import torch
        out = [torch.zeros((70, 90, 4), device="cuda") for _ in range(2)]
        default = gpu_ctx.render_launch()
        gpu_ctx.render(vol, tf, desc, out[0])
        try:
            gpu_ctx.set_render_launch(lv.LAUNCH_GRID, 8, 16)
            gpu_ctx.render(vol, tf, desc, out[1])
        finally:
            gpu_ctx.set_render_launch(**default)
        assert torch.equal(out[0], out[1])
    vol.close()
    tf.close()


def test_unread_voxels_leave_the_ray_alone(gpu_ctx):
    """A sample past a ray's end may map to any table entry: an infinite entry
    that no voxel maps to (values up to 255 of a range to 300) changes nothing."""
    import torch
    import livre_gb300 as lv
    vi = lv.VolumeInformation(192, 64, 1)
    vol = gpu_ctx.blob_volume(vi, 12, 5, 3)
    rgba = lv.linear_ramp_tf(256)
    inf = rgba.copy()
    inf[240:] = np.inf
    mv, proj = lv.orbit_camera(1, 8, vi.world_size, 90, 70, radius_scale=0.8)
    desc = gpu_ctx.render_desc(mv, proj, 90, 70, sse=1.0, data_range=(0.0, 300.0), early_exit=0.7)
    frames = []
    for table in (rgba, inf):
        tf = gpu_ctx.transfer_function(table)
        frames.append(gpu_ctx.render(vol, tf, desc).clone())
        tf.close()
    assert torch.isfinite(frames[0]).all()
    assert torch.equal(frames[0], frames[1])
    vol.close()
