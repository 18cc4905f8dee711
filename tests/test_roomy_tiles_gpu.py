"""uint16 frames whose tile kernel runs with fewer blocks an SM (finest voxels
small on screen) and those that do not: image and sample count equal, bit for
bit, those of the one-thread-per-pixel launch, for the fixed pitches and
another, tables of 16 to 4096 entries, in frames and in batches."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("voxels,block", [(2048, 64), (2048, 128), (768, 96), (256, 64), (2048, 62), (1024, 32)])
@pytest.mark.parametrize("table", [16, 256, 4096])
def test_uint16_frames_bit_identical(native, voxels, block, table):
    import torch
    import livre_gb300 as lv
    ctx = lv.Context(0, pool_bytes=4 << 30)  # every view's bricks stay resident
    voxels = voxels // block * block if block == 62 else voxels
    vi = lv.VolumeInformation(voxels, block, 1, dtype=lv.DT_UINT16)
    vol = ctx.blob_volume(vi, 24, 5, 3)
    tf = ctx.transfer_function(lv.gaussian_peaks_tf(table, seed=6))
    W, H = 641, 479
    items, want = [], []
    for k, radius in enumerate((0.5, 1.0, 3.0)):
        mv, proj = lv.orbit_camera(k, 8, vi.world_size, W, H, radius_scale=radius)
        desc = ctx.render_desc(mv, proj, W, H, sse=2.0, early_exit=0.99)
        ctx.render(vol, tf, desc)
        # one lane per ray, so that the tile kernel renders frames of few rays too
        lv.check(native.lv_test_ray_lanes(ctx.handle, 1, None), ctx.handle)
        img = ctx.render(vol, tf, desc).clone()
        n = ctx.last_stats()
        default = ctx.render_launch()
        try:
            ctx.set_render_launch(lv.LAUNCH_GRID, 8, 16)
            ref = ctx.render(vol, tf, desc).clone()
            m = ctx.last_stats()
        finally:
            ctx.set_render_launch(**default)
            lv.check(native.lv_test_ray_lanes(ctx.handle, 0, None), ctx.handle)
        assert torch.equal(img, ref) and n["n_samples"] == m["n_samples"] > 0 and n["error_flags"] == 0
        items.append((vol, tf, desc, torch.empty_like(img)))
        want.append(ref)
    batch = lv.Batch(ctx)
    batch.render(items)
    torch.cuda.synchronize()
    assert all(torch.equal(i[3], w) for i, w in zip(items, want))
    batch.close()
    vol.close()
    tf.close()
    ctx.close()
