"""Every kernel that shares a ray between lanes: the seven voxel types, both
filters, bricks with and without overlap (clamped taps), 4 and 8 lanes, forced
by lv_test_ray_lanes, against one lane per ray, bit for bit; the typed kernels
against the uint8 one on the same values; and the rule's choices on both sides
of its limits.

Tolerance of the typed comparison: 3e-4 per channel. The densities of the two
volumes differ by the roundings of seven FP32 interpolations, about 2^-21, so a
sample's colour by less than 1e-6 and a ray of at most 300 samples by less than
3e-4."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# lv_dtype, numpy type, value map of a byte, data range
TYPES = {"u8": (1, np.uint8, lambda v: v, (0.0, 255.0)),
         "u16": (2, np.uint16, lambda v: v.astype(np.int64) * 257, (0.0, 65535.0)),
         "i8": (4, np.int8, lambda v: v.astype(np.int16) - 128, (-128.0, 127.0)),
         "i16": (5, np.int16, lambda v: v.astype(np.int32) * 100 - 12000, (-12000.0, 13500.0)),
         "u32": (3, np.uint32, lambda v: v.astype(np.uint64) * 16777, (0.0, 255.0 * 16777)),
         "i32": (6, np.int32, lambda v: v.astype(np.int64) * 1000 - 100000, (-100000.0, 155000.0)),
         "f32": (0, np.float32, lambda v: v.astype(np.float64) / 255.0 * 3.5 - 1.0, (-1.0, 2.5))}


def byte_field(n):
    """Smooth bodies and noise as bytes (z, y, x)."""
    g = np.mgrid[0:n, 0:n, 0:n].astype(np.float64) / n
    r = np.random.default_rng(5)
    v = 0.1 * r.random((n, n, n))
    for c in r.uniform(0.2, 0.8, (5, 3)):
        v += 0.8 * np.exp(-((g[0] - c[0]) ** 2 + (g[1] - c[1]) ** 2 + (g[2] - c[2]) ** 2) / 0.02)
    return (np.clip(v, 0, 1) * 255).astype(np.uint8)


def volume(ctx, lv, name, n, block, overlap):
    """The finest level of an n^3 volume of that type, loaded."""
    dtype, ntype, vmap, _ = TYPES[name]
    vi = lv.VolumeInformation(n, block, overlap, dtype=dtype)
    level, side = vi.depth - 1, n // block
    padded = np.pad(vmap(byte_field(n)).astype(ntype), overlap, mode="edge")
    size = block + 2 * overlap
    bricks = {int(lv.NodeId(level, (x, y, z))): np.ascontiguousarray(
        padded[z * block:z * block + size, y * block:y * block + size, x * block:x * block + size])
        for z in range(side) for y in range(side) for x in range(side)}

    def get_data(node_id, dst, nbytes):
        b = bricks.get(node_id)
        if b is None or b.nbytes != nbytes:
            return False
        C.memmove(dst, b.ctypes.data, nbytes)
        return True

    vol = ctx.callback_volume(vi, get_data)
    vol.load(sorted(bricks))
    return vi, vol


def cast(ctx, lv, native, vol, tf, desc, lanes):
    """Image, samples and lanes of a frame with that many lanes per ray (0: the rule's)."""
    last = C.c_uint32()
    try:
        lv.check(native.lv_test_ray_lanes(ctx.handle, lanes, None), ctx.handle)
        img = ctx.render(vol, tf, desc).clone()
        st = ctx.last_stats()
    finally:
        lv.check(native.lv_test_ray_lanes(ctx.handle, 0, C.byref(last)), ctx.handle)
    assert st["error_flags"] == 0
    return img, st["n_samples"], last.value


@pytest.mark.parametrize("name", sorted(TYPES))
@pytest.mark.parametrize("block,overlap", [(16, 0), (16, 1), (24, 2), (64, 1)])
@pytest.mark.parametrize("filt", [0, 1])
def test_lanes_bit_identical(gpu_ctx, native, name, block, overlap, filt):
    import torch
    import livre_gb300 as lv
    n = 4 * block if block < 64 else 128
    vi, vol = volume(gpu_ctx, lv, name, n, block, overlap)
    tf = gpu_ctx.transfer_function(lv.gaussian_peaks_tf(64, seed=6))
    taken = 0
    for k, (W, H) in enumerate([(1, 1), (5, 7), (33, 17), (121, 117)]):
        mv, proj = lv.orbit_camera(k, 8, vi.world_size, W, H, radius_scale=0.9)
        for early in (0.6, 2.0):
            desc = gpu_ctx.render_desc(mv, proj, W, H, sse=1.0, min_lod=vi.depth - 1, filt=filt, early_exit=early,
                                       data_range=TYPES[name][3])
            ref, samples, one = cast(gpu_ctx, lv, native, vol, tf, desc, 1)
            assert one == 1
            for lanes in (4, 8):
                img, m, used = cast(gpu_ctx, lv, native, vol, tf, desc, lanes)
                assert used == lanes and m == samples and torch.equal(img, ref)
            taken += samples
    assert taken > 10000
    vol.close()
    tf.close()


@pytest.mark.parametrize("name", sorted(set(TYPES) - {"u8"}))
@pytest.mark.parametrize("overlap", [0, 1])
@pytest.mark.parametrize("filt", [0, 1])
def test_types_equal_the_uint8_kernel(gpu_ctx, native, name, overlap, filt):
    import livre_gb300 as lv
    tf = gpu_ctx.transfer_function(lv.linear_ramp_tf(64))
    frames = {}
    for t in ("u8", name):
        vi, vol = volume(gpu_ctx, lv, t, 64, 16, overlap)
        mv, proj = lv.orbit_camera(3, 8, vi.world_size, 97, 61, radius_scale=1.0)
        # no early termination: the two volumes take the same samples
        desc = gpu_ctx.render_desc(mv, proj, 97, 61, sse=1.0, min_lod=vi.depth - 1, filt=filt, early_exit=2.0,
                                   data_range=TYPES[t][3], samples_per_ray=200)
        frames[t] = [cast(gpu_ctx, lv, native, vol, tf, desc, lanes) for lanes in (1, 4, 8)]
        vol.close()
    for a, b in zip(frames["u8"], frames[name]):
        assert a[1] == b[1] > 1000
        assert float((a[0] - b[0]).abs().max()) <= 3e-4
    tf.close()


# sizes of 16:9 viewports whose candidate rays go past every limit of the rule
WIDTHS = [64, 160, 320, 480, 640, 960, 1280, 1920, 2560]


@pytest.mark.parametrize("name,overlap,filt", [("u8", 1, 1), ("u16", 1, 1), ("i8", 1, 1), ("i16", 1, 1), ("f32", 1, 1),
                                               ("u8", 0, 1), ("u16", 0, 1), ("f32", 0, 1), ("u8", 1, 0), ("u16", 0, 0)])
def test_both_sides_of_the_rule(gpu_ctx, native, name, overlap, filt):
    import torch
    import livre_gb300 as lv
    vi, vol = volume(gpu_ctx, lv, name, 64, 16, overlap)
    tf = gpu_ctx.transfer_function(lv.gaussian_peaks_tf(64, seed=6))
    lanes = []
    for W in WIDTHS:
        H = W * 9 // 16
        mv, proj = lv.orbit_camera(2, 8, vi.world_size, W, H, radius_scale=0.8)
        desc = gpu_ctx.render_desc(mv, proj, W, H, sse=1.0, min_lod=vi.depth - 1, filt=filt, data_range=TYPES[name][3],
                                   early_exit=0.99)
        img, samples, used = cast(gpu_ctx, lv, native, vol, tf, desc, 0)
        ref, want, _ = cast(gpu_ctx, lv, native, vol, tf, desc, 1)
        assert samples == want > 0 and torch.equal(img, ref)
        lanes.append(used)
    assert lanes == sorted(lanes, reverse=True) and set(lanes) == {1, 4, 8}
    vol.close()
    tf.close()
