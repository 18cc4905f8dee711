"""The clear before a frame covers the leaf grid of a deep octree at the GPU's
rate whatever the rect: a frame of one row takes no longer than one of a
thousand rows, although it has few pixels to clear."""
import time

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("voxels", [8192, (8192, 2016, 4000)])
def test_narrow_rects_of_a_deep_octree(gpu_ctx, voxels):
    import torch
    import livre_gb300 as lv
    vi = lv.VolumeInformation(voxels, 32, 1)  # up to 256^3 leaf cells
    vol = gpu_ctx.blob_volume(vi, 4, 3)
    tf = gpu_ctx.transfer_function(lv.linear_ramp_tf(64))
    W, H = 1024, 1024
    # the volume is beside the frustum: every pixel is cleared only
    mv, proj = lv.look_at((0.0, 0.0, 6.0), (6.0, 0.0, 0.0)), lv.perspective(40.0, 1.0, 0.1, 50.0)
    out = torch.empty((H, W, 4), device="cuda")

    def frame_us(rect):
        desc = gpu_ctx.render_desc(mv, proj, W, H, sse=8.0, rect=rect)
        times = []
        for _ in range(24):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            gpu_ctx.render(vol, tf, desc, out)
            torch.cuda.synchronize()
            times.append((time.perf_counter() - t0) * 1e6)
        return sorted(times)[len(times) // 2]

    whole = frame_us((0, 0, W, H))
    for rect in ((0, 0, 256, 1), (3, 5, 8, 20), (0, 0, 1, 1024)):
        assert frame_us(rect) < 1.5 * whole
    # and the grid is cleared whole: the same frame before and after
    mv, p = lv.orbit_camera(1, 8, vi.world_size, 96, 64, radius_scale=1.5)
    desc = gpu_ctx.render_desc(mv, p, 96, 64, sse=8.0)
    first = gpu_ctx.render(vol, tf, desc).clone()
    gpu_ctx.render(vol, tf, gpu_ctx.render_desc(mv, p, 96, 64, sse=16.0))
    assert torch.equal(gpu_ctx.render(vol, tf, desc), first)
    vol.close()
    tf.close()
