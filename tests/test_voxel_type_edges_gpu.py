"""Every voxel type's kernel with clamped edges (bricks without overlap) and
with and without look-ahead, against the oracle. The volumes hold a uint8
volume's bricks under an affine map, as in test_voxel_types_gpu.py.

Tolerance: max per-channel |GPU - oracle| <= 1/255, the ray cast's own bar.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TYPES = [
    (4, np.int8, lambda v: v.astype(np.int16) - 128, (-128.0, 127.0)),
    (5, np.int16, lambda v: v.astype(np.int32) * 100 - 12000, (-12000.0, 13500.0)),
    (3, np.uint32, lambda v: v.astype(np.uint64) * 16777, (0.0, 255.0 * 16777)),
    (6, np.int32, lambda v: v.astype(np.int64) * 1000 - 100000, (-100000.0, 155000.0)),
    (0, np.float32, lambda v: v.astype(np.float64) / 255.0 * 3.5 - 1.0, (-1.0, 2.5)),
]


@pytest.mark.parametrize("dtype,ntype,vmap,rng", TYPES)
@pytest.mark.parametrize("filt,lookahead", [(0, 0), (1, 1), (1, 0)])
def test_clamped_edges(gpu_ctx, oracle, dtype, ntype, vmap, rng, filt, lookahead):
    import livre_gb300 as lv
    vi = lv.VolumeInformation(64, 16, 0, dtype=dtype)
    ovol = oracle.volume(64, 16, 0)
    bp = oracle.blob_params(6, 3, 0, 1)
    bricks = {n.id: np.ascontiguousarray(vmap(oracle.blob_brick(ovol, bp, n.id)).astype(ntype))
              for n in vi.all_nodes()}

    def get_data(node_id, dst, nbytes):
        b = bricks.get(node_id)
        if b is None or b.nbytes != nbytes:
            return False
        C.memmove(dst, b.ctypes.data, nbytes)
        return True

    vol = gpu_ctx.callback_volume(vi, get_data)
    tf_rgba = lv.linear_ramp_tf(64)
    tf = gpu_ctx.transfer_function(tf_rgba)
    W, H = 37, 29
    default = gpu_ctx.render_launch()
    try:
        gpu_ctx.set_render_launch(**dict(default, lookahead=lookahead))
        mv, proj = lv.orbit_camera(3, 8, vi.world_size, W, H, radius_scale=1.2)
        desc = gpu_ctx.render_desc(mv, proj, W, H, sse=1.0, filt=filt, data_range=rng)
        img = gpu_ctx.render(vol, tf, desc).cpu().numpy()
        st = gpu_ctx.last_stats()
    finally:
        gpu_ctx.set_render_launch(**default)
    assert st["error_flags"] == 0
    ids, _ = oracle.select_visible(ovol, mv, proj, H, 1.0)
    view = oracle.make_view(mv, proj, W, H, st["samples_per_ray"], filt=filt, range_lo=rng[0],
                            range_hi=rng[1])
    ref, ns = oracle.raycast(ovol, dtype, ids, np.stack([bricks[int(i)] for i in ids]), tf_rgba, view)
    assert ns > 500
    # the nearest filter reads another voxel where FP32 and FP64 positions
    # fall on two sides of a voxel face: a few pixels of a frame
    off = np.abs(img - ref).max(-1) > 1.0 / 255.0
    assert off.sum() <= (2 if filt == 0 else 0), off.sum()
    vol.close()
    tf.close()
