"""Every voxel type's kernel with clamped edges (bricks without overlap) and
with and without look-ahead, against the uint8 kernel on the same values: the
volumes hold a uint8 volume's bricks under an affine map, with the data range
mapped the same way. (Not against the oracle: without overlap the trilinear
filter jumps at brick faces, where FP32 and FP64 positions fall on two
sides.)

Tolerance: 1/255 per channel. The densities of the mapped volume and of the
uint8 one differ by the roundings of seven FP32 interpolations, about 2^-21,
so a sample's colour by less than 1e-6 and a ray of at most 300 samples by
less than 3e-4.
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


def frame(ctx, lv, oracle, dtype, ntype, vmap, rng, filt, lookahead):
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

    vol = ctx.callback_volume(vi, get_data)
    tf = ctx.transfer_function(lv.linear_ramp_tf(64))
    W, H = 37, 29
    default = ctx.render_launch()
    try:
        ctx.set_render_launch(**dict(default, lookahead=lookahead))
        mv, proj = lv.orbit_camera(3, 8, vi.world_size, W, H, radius_scale=1.2)
        # no early termination: the two volumes take the same samples
        desc = ctx.render_desc(mv, proj, W, H, sse=1.0, filt=filt, data_range=rng, early_exit=2.0)
        img = ctx.render(vol, tf, desc).cpu().numpy()
        st = ctx.last_stats()
    finally:
        ctx.set_render_launch(**default)
    assert st["error_flags"] == 0 and st["n_samples"] > 500
    vol.close()
    tf.close()
    return img, st["n_samples"]


@pytest.mark.parametrize("dtype,ntype,vmap,rng", TYPES)
@pytest.mark.parametrize("filt,lookahead", [(0, 0), (1, 1), (1, 0)])
def test_clamped_edges(gpu_ctx, oracle, dtype, ntype, vmap, rng, filt, lookahead):
    import livre_gb300 as lv
    img, n = frame(gpu_ctx, lv, oracle, dtype, ntype, vmap, rng, filt, lookahead)
    ref, n_ref = frame(gpu_ctx, lv, oracle, lv.DT_UINT8, np.uint8, lambda v: v, (0.0, 255.0), filt, lookahead)
    assert n == n_ref
    assert np.abs(img - ref).max() <= 1.0 / 255.0
