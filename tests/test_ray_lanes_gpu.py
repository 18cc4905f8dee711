"""The rule of the lanes per ray: where it shares rays the frame is not slower
than with one lane per ray, in views where limits on rays and pixels per voxel
alone shared them at a loss of 11 to 20 %."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

# voxels, block, overlap, dtype (lv_dtype), viewport, LOD px, camera, table
CASES = [(1024, 128, 1, 2, (1600, 1200), 2.0, 1.6, 4096), (256, 32, 1, 2, (1280, 960), 1.0, 1.6, 256),
         (1024, 64, 1, 2, (800, 600), 1.0, None, 256)]


@pytest.mark.parametrize("voxels,block,overlap,dtype,size,sse,radius,table", CASES)
def test_sharing_rays_does_not_slow_a_frame(native, voxels, block, overlap, dtype, size, sse, radius, table):
    import torch
    import livre_gb300 as lv
    ctx = lv.Context(0, pool_bytes=6 << 30)
    vi = lv.VolumeInformation(voxels, block, overlap, dtype=dtype)
    vol = ctx.fbm_volume(vi, 3)
    tf = ctx.transfer_function(lv.gaussian_peaks_tf(table, seed=12))
    W, H = size
    if radius is None:  # inside, looking along the volume
        mv, proj = lv.look_at((-0.2, -0.13, -0.37), (0.35, 0.25, 0.55)), lv.perspective(45.0, W / H, 0.01, 15.0)
    else:
        mv, proj = lv.orbit_camera(5, 64, vi.world_size, W, H, radius_scale=radius)
    desc = ctx.render_desc(mv, proj, W, H, sse=sse, early_exit=0.99, step_policy=lv.STEP_REFERENCE)
    out = torch.empty((H, W, 4), device="cuda")
    ms, images, last = {}, {}, C.c_uint32()
    for lanes in (1, 0, 1, 0):
        lv.check(native.lv_test_ray_lanes(ctx.handle, lanes, None), ctx.handle)
        times = []
        for _ in range(9):
            ctx.render(vol, tf, desc, out)
            torch.cuda.synchronize()
            times.append(ctx.last_stats()["raycast_ms"])
        ms[lanes] = min(min(times), ms.get(lanes, 1e9))
        images[lanes] = out.clone()
    lv.check(native.lv_test_ray_lanes(ctx.handle, 0, C.byref(last)), ctx.handle)
    assert torch.equal(images[0], images[1]) and ctx.last_stats()["n_samples"] > 0
    assert last.value in (1, 4, 8)
    assert ms[0] < 1.08 * ms[1]
    vol.close()
    tf.close()
    ctx.close()


def test_lanes_hook_rejects_other_counts(gpu_ctx, native):
    import livre_gb300 as lv
    from livre_gb300 import _abi
    for lanes in (2, 3, 16):
        assert native.lv_test_ray_lanes(gpu_ctx.handle, lanes, None) == _abi.LV_EINVAL
    lv.check(native.lv_test_ray_lanes(gpu_ctx.handle, 0, None), gpu_ctx.handle)
