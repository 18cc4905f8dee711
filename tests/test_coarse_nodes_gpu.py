"""Frames whose rendered nodes cover many cells of the leaf grid: the nodes of
one level alone (rows of 8 to 64 cells, octrees with unequal sides), whose
samples are counted, and a view of an 8192^3 octree that shows only its root."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("voxels,block", [(1024, 16), ((1024, 256, 500), 16), ((40, 640, 160), 16)])
@pytest.mark.parametrize("sync", [True, False])
def test_nodes_of_each_level(gpu_ctx, voxels, block, sync):
    """Every sample inside the octree finds its brick: the grid has no hole. A
    row of cells left out would be 1/64 of the samples at least; a sample on a
    face may fall either way, far below the 1/200 allowed."""
    import torch
    import livre_gb300 as lv
    vi = lv.VolumeInformation(voxels, block, 1)
    vol = gpu_ctx.blob_volume(vi, 12, 5)
    tf = gpu_ctx.transfer_function(lv.gaussian_peaks_tf(64, seed=2))
    W, H = 96, 80
    for level in range(vi.depth):
        if level > 3:
            break
        mv, proj = lv.orbit_camera(level, 8, vi.world_size, W, H, radius_scale=1.1)
        frames, counts = [], []
        for launch in (None, (lv.LAUNCH_GRID, 8, 16)):
            default = gpu_ctx.render_launch()
            desc = gpu_ctx.render_desc(mv, proj, W, H, sse=1e-6, min_lod=0, max_lod=level, samples_per_ray=300, early_exit=2.0,
                                       synchronous=sync, max_uploads=1 << 20)
            try:
                if launch:
                    gpu_ctx.set_render_launch(*launch)
                for _ in range(3):
                    frame = gpu_ctx.render(vol, tf, desc).clone()
                st = gpu_ctx.last_stats()
            finally:
                gpu_ctx.set_render_launch(**default)
            frames.append(frame)
            counts.append(st["n_samples"])
            assert st["error_flags"] == 0 and st["max_level"] == level
        assert torch.equal(frames[0], frames[1]) and counts[0] == counts[1] > 0
        full = expected_samples(vi, mv, proj, W, H, 300)
        assert abs(counts[0] - full) <= full / 200
    vol.close()
    tf.close()


def expected_samples(vi, mv, proj, W, H, n):
    """Samples of all rays inside the octree's leaf cells, in double precision."""
    m = np.asarray(mv, np.float64).reshape(4, 4).T
    p = np.asarray(proj, np.float64).reshape(4, 4).T
    im, ip = np.linalg.inv(m), np.linalg.inv(p)
    nx, ny = (np.arange(W) + 0.5) * 2 / W - 1, (np.arange(H) + 0.5) * 2 / H - 1
    c = np.stack([np.broadcast_to(nx[None, :], (H, W)), np.broadcast_to(ny[:, None], (H, W)),
                  np.full((H, W), -1.0), np.ones((H, W))], -1)
    e = c @ ip.T
    e = e[..., :3] / e[..., 3:]
    eye = im[:3, 3]
    d = e @ im[:3, :3].T
    d /= np.linalg.norm(d, axis=-1, keepdims=True)
    half = np.array(vi.world_size) / 2
    with np.errstate(divide="ignore"):
        a, b = (-half - eye) / d, (half - eye) / d
    t0, t1 = np.minimum(a, b).max(-1), np.maximum(a, b).min(-1)
    near = p[2, 3] / (p[2, 2] - 1.0)
    tlo = np.maximum(t0, -near / (e[..., 2] / np.linalg.norm(e, axis=-1)))
    total = 0
    dims = np.array([r << (vi.depth - 1) for r in vi.root_blocks])
    cell = np.array(vi.world_size) / dims.max()
    k = np.arange(2 * n)[:, None]
    for y in range(H):
        hit = t0[y] <= t1[y]
        t = t0[y] + k / n
        inside = hit & (t >= tlo[y]) & (t < t1[y])
        pos = eye + d[y][None] * t[..., None]
        total += int((inside & ((pos + half) / cell <= dims + 1e-9).all(-1)).sum())
    return total


@pytest.mark.parametrize("sync", [True, False])
def test_a_view_of_the_root_alone(gpu_ctx, sync):
    import torch
    import livre_gb300 as lv
    vi = lv.VolumeInformation(8192, 32, 1)  # 256^3 leaf cells under the root
    vol = gpu_ctx.blob_volume(vi, 12, 5)
    tf = gpu_ctx.transfer_function(lv.linear_ramp_tf(64))
    mv, proj = lv.orbit_camera(1, 8, vi.world_size, 256, 256, radius_scale=8.0)
    gpu_ctx.render(vol, tf, gpu_ctx.render_desc(mv, proj, 256, 256, sse=32.0))
    desc = gpu_ctx.render_desc(mv, proj, 256, 256, sse=32.0, synchronous=sync)
    times = []
    for _ in range(12):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        gpu_ctx.render(vol, tf, desc)
        torch.cuda.synchronize()
        times.append((time.perf_counter() - t0) * 1e3)
    st = gpu_ctx.last_stats()
    assert st["n_rendered"] == 1 and st["max_level"] == 0 and st["n_samples"] > 0
    # the GPU's warps share the cells: a single one takes 25 ms
    assert sorted(times)[len(times) // 2] < 10.0
    vol.close()
    tf.close()
