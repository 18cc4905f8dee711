"""The one-launch residency pass of lv_render (lookup, ancestor fallback, leaf
grid) against the batch's three launches, on volumes of which a random part is
resident: the same image bit for bit and the same counts. Resident sets from
nothing (every node missing) over coarse levels only to everything; octrees
with several root blocks, one level, and one brick."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("voxels,block", [((128, 128, 128), 16), ((128, 96, 64), 16), ((64, 64, 64), 32),
                                          ((20, 20, 20), 20), ((300, 16, 16), 16)])
@pytest.mark.parametrize("share", [0.0, 0.2, 0.6, 1.0])
def test_partly_resident_frames_match_the_batch(gpu_ctx, voxels, block, share):
    import torch
    import livre_gb300 as lv
    vi = lv.VolumeInformation(voxels, block, 1)
    vol = gpu_ctx.blob_volume(vi, 10, 4, 5)
    tf = gpu_ctx.transfer_function(lv.linear_ramp_tf(64))
    rng = np.random.default_rng(int(share * 10) + block)
    nodes = [n.id for n in vi.all_nodes()]
    resident = [i for i in nodes if rng.random() < share]
    if resident:
        vol.load(resident)
    batch = lv.Batch(gpu_ctx)
    W, H = 61, 47
    for k, sse in ((0, 0.5), (3, 3.0), (5, 8.0)):
        mv, proj = lv.orbit_camera(k, 8, vi.world_size, W, H, radius_scale=1.1)
        desc = gpu_ctx.render_desc(mv, proj, W, H, sse=sse, synchronous=False, max_uploads=0)
        img = gpu_ctx.render(vol, tf, desc)
        st = gpu_ctx.last_stats()
        out = torch.empty_like(img)
        batch.render([(vol, tf, desc, out)])
        bt = batch.stats(1)[0][0]
        assert torch.equal(img, out)
        for f in ("n_visible", "n_visited", "n_rendered", "n_available", "n_not_available", "max_level",
                  "samples_per_ray", "n_samples", "error_flags"):
            assert st[f] == bt[f], f
        assert st["n_available"] + st["n_not_available"] == st["n_visible"]
        if share == 1.0:
            # the synchronous form of the pass on the same bricks
            ds = gpu_ctx.render_desc(mv, proj, W, H, sse=sse)
            assert torch.equal(gpu_ctx.render(vol, tf, ds), img)
            ss = gpu_ctx.last_stats()
            assert ss["n_uploaded"] == 0 and ss["n_rendered"] == st["n_rendered"]
    batch.close()
    vol.close()
    tf.close()
