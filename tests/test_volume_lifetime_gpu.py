"""A volume is destroyed as soon as its last request is collected, or while a
batch still remembers its misses: nothing touches it afterwards, and the bricks
it pinned are given back."""
import pytest

pytestmark = pytest.mark.gpu


def view(ctx, lv, vi, W=64, H=48, **kw):
    mv, proj = lv.orbit_camera(1, 8, vi.world_size, W, H, radius_scale=1.2)
    return ctx.render_desc(mv, proj, W, H, sse=1.0, **kw)


def test_volume_destroyed_right_after_its_last_request():
    import torch
    import livre_gb300 as lv
    vi = lv.VolumeInformation(128, 32, 1)
    # 16 slots for 8 visible bricks: bricks left pinned would keep later volumes out
    ctx = lv.Context(0, pool_bytes=640 << 10)
    tf = ctx.transfer_function(lv.linear_ramp_tf(64))
    first = ctx.blob_volume(vi, 8, 3)
    server = lv.Server(ctx)
    out = [torch.empty((48, 64, 4), device="cuda") for _ in range(3)]
    ref = None
    for k in range(40):
        vol = first if k == 0 else ctx.blob_volume(vi, 8, 3)
        tickets = [server.submit(vol, tf, view(ctx, lv, vi), o) for o in out]
        results = [server.wait(t) for t in tickets]
        vol.close()
        assert all(r["status"] == 0 and r["stats"]["n_samples"] > 0 for r in results)
        ref = out[0].clone() if ref is None else ref
        assert all(torch.equal(o, ref) for o in out)
    assert server.counters()["completed"] == 120
    server.close()
    ctx.close()


def test_batch_forgets_the_misses_of_a_destroyed_volume(gpu_ctx):
    import torch
    import livre_gb300 as lv
    vi = lv.VolumeInformation(128, 32, 1)
    tf = gpu_ctx.transfer_function(lv.linear_ramp_tf(64))
    batch = lv.Batch(gpu_ctx)
    keep = gpu_ctx.blob_volume(vi, 8, 3)
    outs = [torch.empty((48, 64, 4), device="cuda") for _ in range(2)]
    for seed in range(4):
        gone = gpu_ctx.blob_volume(vi, 8, 10 + seed)
        items = [(v, tf, view(gpu_ctx, lv, vi, synchronous=False, max_uploads=64), o)
                 for v, o in zip((gone, keep), outs)]
        batch.render(items)  # every brick of `gone` misses
        gone.close()
        batch.render(items[1:])
        torch.cuda.synchronize()
        resident = set(keep.resident())
        assert len(resident) == len(keep.resident()) > 0
    assert batch.stats(1)[0][0]["error_flags"] == 0
    batch.close()
    keep.close()
    tf.close()
