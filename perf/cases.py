"""The work a user of livre_gb300 has it do, as cases that can be timed and compared.

A case is a dict of plain values. `prepare` makes what a program holds before the call (a
context with its brick pool, volumes, transfer functions, a batch or a server, a camera),
`run` makes one pass through the public Python entry points, `exact` gives the same result in
64 bits where a volume made here allows it.

Kinds:
  frame      one view of a resident volume: `Context.render`
  cold       one view with an empty brick pool: `Context.purge`, then `Context.render`
             streams every visible brick
  batch      many views in one `Batch.render`
  serve      a burst of requests through a `Server`
  histogram  value histograms of bricks: `Volume.histogram`
  select     level-of-detail selection alone: `Context.select_visible`

Volume sources: `field` (made here on the GPU, handed over brick by brick through a data-source
callback), `blob` and `blob_host` (the framework's Gaussian blobs, generated on the device or
kept in page-locked host memory), `fbm` (the framework's fractal noise, generated on a miss).
"""
import ctypes
import math

import numpy as np
import torch

import livre_gb300 as lv

GIB = 1 << 30
DTYPES = {"u8": lv.DT_UINT8, "u16": lv.DT_UINT16, "i8": lv._abi.DT_INT8, "i16": lv._abi.DT_INT16, "f32": lv._abi.DT_FLOAT}
BYTES = {"u8": 1, "u16": 2, "i8": 1, "i16": 2, "f32": 4}
TORCH = {"u8": torch.uint8, "i8": torch.int8, "i16": torch.int16, "f32": torch.float32}
# values of the made volumes, and the range the transfer function spans
VALUES = {"u8": (0.0, 255.0), "i8": (0.0, 127.0), "i16": (-1000.0, 3000.0), "f32": (0.0, 1.0)}


# ------------------------------------------------------------------ cases
def listed():
    frame = dict(kind="frame", overlap=1, filter="trilinear", step="half_voxel", camera="orbit", radius=2.5,
                 sync=True)
    return [
        # a thumbnail of a small CT-like volume with odd sizes (a file browser, a picker): latency
        dict(frame, name="preview_i16_100", source="field", voxels="100x90x75", block=32, dtype="i16",
             width=129, height=97, sse=1.0, early=0.999, tf="ramp", tf_n=256, min_lod=2),
        # the plain workload: a small uint8 volume in 32^3 bricks, 512 x 512
        dict(frame, name="frame_u8_256", source="field", voxels="256x256x256", block=32, dtype="u8",
             width=512, height=512, sse=1.0, early=0.999, tf="ramp", tf_n=256, min_lod=3),
        # the plain workload at scale: 2048^3 uint8 in 64^3 bricks at 1080p, bricks resident
        dict(frame, name="frame_u8_2048", source="blob", blobs=256, noise=8, voxels="2048x2048x2048", block=64,
             dtype="u8", width=1920, height=1080, sse=2.0, early=0.99, tf="peaks", tf_n=256, min_lod=0),
        # inside a uint16 volume in 128^3 bricks, 4K, the reference's step rule, 4096-entry table
        dict(frame, name="frame_u16_inside_4k", source="fbm", voxels="2048x2048x2048", block=128, dtype="u16",
             width=3840, height=2160, sse=2.0, early=0.999, tf="peaks", tf_n=4096, step="reference",
             camera="inside", min_lod=0),
        # a simulation's float32 field with ragged extents, an odd viewport
        dict(frame, name="frame_f32_ragged", source="field", voxels="380x333x290", block=48, dtype="f32",
             width=1001, height=701, sse=1.0, early=0.99, tf="peaks", tf_n=512, radius=1.6, min_lod=3),
        # the reference's default settings: nearest filter, its step rule, its default table, no
        # overlap, asynchronous frames
        dict(frame, name="frame_u8_nearest", source="field", voxels="512x512x512", block=64, overlap=0, dtype="u8",
             width=1024, height=768, sse=4.0, early=0.999, tf="default", tf_n=256, filter="nearest",
             step="reference", radius=1.5, sync=False, min_lod=3),
        # the first frame of a data set kept in host memory: every visible brick streams
        dict(frame, name="cold_u8_host", kind="cold", source="blob_host", blobs=48, noise=4, voxels="512x512x512",
             block=64, dtype="u8", width=1280, height=720, sse=1.0, early=0.99, tf="peaks", tf_n=256, radius=1.4,
             min_lod=0),
        # the first frame of an out-of-core fly-through: bricks made when they miss
        dict(frame, name="cold_u16_fbm", kind="cold", source="fbm", voxels="1024x1024x1024", block=128,
             dtype="u16", width=1920, height=1080, sse=2.0, early=0.999, tf="peaks", tf_n=4096, step="reference",
             camera="inside", min_lod=0),
        # many users' views of several volumes in one batch, mixed sizes
        dict(name="batch_mixed_24", kind="batch", views=24, sizes="mixed"),
        # a burst of requests at a render server
        dict(name="serve_burst_12", kind="serve", views=12, sizes="small"),
        # the histogram of a whole data set at its finest level, per brick too
        dict(name="histogram_u8_512", kind="histogram", source="field", voxels="512x512x512", block=64, overlap=1,
             dtype="u8", bins=256),
        # selection in a deep octree, the camera inside it
        dict(name="select_8192", kind="select", voxels="8192x8192x8192", block=64, overlap=1, dtype="u8",
             width=1920, height=1080, sse=1.0, camera="inside", radius=1.5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cube(n):
    return "%dx%dx%d" % (n, n, n)


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "cold", "batch", "serve", "histogram", "select"])
    if kind in ("batch", "serve"):
        return dict(kind=kind, views=rng.randint(2, 24 if kind == "batch" else 16), sizes=rng.choice(["small", "mixed"]))
    if kind == "select":
        block = rng.choice([32, 64, 128])
        return dict(kind=kind, voxels=_cube(_log(rng, 256, 64 * block if block == 32 else 8192)), block=block, overlap=1, dtype="u8",
                    width=_log(rng, 128, 1920), height=_log(rng, 96, 1080), sse=round(rng.uniform(1.0, 8.0), 2),
                    camera=rng.choice(["inside", "orbit"]), radius=round(rng.uniform(0.6, 2.5), 2))
    if kind == "histogram":
        return dict(kind=kind, source="field", voxels="x".join(str(_log(rng, 96, 400)) for _ in range(3)),
                    block=rng.choice([30, 32, 48, 64]), overlap=rng.choice([0, 1, 2]),
                    dtype=rng.choice(["u8", "i16", "f32"]), bins=rng.choice([64, 100, 256, 1024]))
    c = dict(kind=kind, filter="trilinear", step=rng.choice(["half_voxel", "reference"]), camera="orbit",
             radius=round(rng.uniform(1.2, 2.5), 2), sync=True, width=_log(rng, 96, 2560), height=_log(rng, 64, 1440),
             sse=round(rng.uniform(1.0, 4.0), 2), early=rng.choice([0.99, 0.999]),
             tf=rng.choice(["ramp", "peaks", "default"]), min_lod=0, overlap=1)
    c["tf_n"] = 256 if c["tf"] == "default" else rng.choice([64, 256, 1000, 4096])
    source = "blob_host" if kind == "cold" else rng.choice(["field", "field", "field", "blob", "fbm"])
    c["source"] = source
    if source == "field":
        c["voxels"] = "x".join(str(_log(rng, 64, 384)) for _ in range(3))
        c["block"] = rng.choice([24, 30, 32, 48, 64])
        c["dtype"] = rng.choice(["u8", "u8", "i8", "i16", "f32"])
        c["overlap"] = rng.choice([0, 1, 1, 1, 2])
        c["filter"] = rng.choice(["trilinear", "trilinear", "nearest"])
        c["sync"] = rng.choice([True, True, False])
        c["min_lod"] = _info(c).depth - 1
    elif source == "fbm":
        c.update(voxels=_cube(rng.choice([512, 1024])), block=rng.choice([64, 128]), dtype=rng.choice(["u8", "u16"]),
                 camera=rng.choice(["inside", "orbit"]))
    else:
        c.update(voxels=_cube(rng.choice([256, 512] if kind == "cold" else [256, 512, 1024])), block=rng.choice([32, 64]),
                 dtype=rng.choice(["u8", "u16"]), blobs=rng.randint(16, 96), noise=rng.choice([0, 4, 8]))
    return c


def _voxels(case):
    return [int(n) for n in case["voxels"].split("x")]


def _info(case):
    return lv.VolumeInformation(_voxels(case), case["block"], case["overlap"], dtype=DTYPES[case["dtype"]])


# ---------------------------------------------------------------- volumes
def _field(case, seed):
    """The finest level of a made volume as a (z, y, x) tensor over whole bricks: bright smooth
    bodies on a dark, slightly noisy ground, as in a stained or scanned specimen."""
    vi = _info(case)
    B, L = vi.block_size, vi.depth - 1
    n = [(vi.root_blocks[a] << L) * B[a] for a in range(3)]
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    v = 0.03 + 0.02 * torch.rand((n[2], n[1], n[0]), generator=g, device=dev)
    r = np.random.default_rng(seed)
    side = max(n)
    for _ in range(24):
        c = [r.uniform(0.1, 0.9) * n[a] for a in range(3)]
        s = r.uniform(0.02, 0.09) * side
        amp = r.uniform(0.2, 0.9)
        lo = [max(0, int(c[a] - 3.5 * s)) for a in range(3)]
        hi = [min(n[a], int(c[a] + 3.5 * s) + 1) for a in range(3)]
        e = [torch.exp(-((torch.arange(lo[a], hi[a], device=dev, dtype=torch.float32) - c[a]) / s) ** 2 / 2) for a in range(3)]
        v[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]] += amp * e[2][:, None, None] * e[1][None, :, None] * e[0][None, None, :]
    lo, hi = VALUES[case["dtype"]]
    v = v.clamp_(0, 1) * (hi - lo) + lo
    return v if case["dtype"] == "f32" else v.floor_().to(TORCH[case["dtype"]])


def _padded(v, vi):
    """Repeats the border voxels `overlap` times on every side, as a data source fills them."""
    for a in range(3):
        o = vi.overlap[2 - a]
        if o:
            i = torch.arange(-o, v.shape[a] + o, device=v.device).clamp_(0, v.shape[a] - 1)
            v = v.index_select(a, i)
    return v


def _cut(v, vi, level):
    """{node id: brick} of one level's voxels."""
    p, N, B = _padded(v, vi), vi.max_block, vi.block_size
    bricks = p.unfold(0, N[2], B[2]).unfold(1, N[1], B[1]).unfold(2, N[0], B[0]).contiguous().cpu().numpy()
    return {int(lv.NodeId(level, (x, y, z))): bricks[z, y, x]
            for z in range(bricks.shape[0]) for y in range(bricks.shape[1]) for x in range(bricks.shape[2])}


def _volume(ctx, case, seed):
    vi = _info(case)
    if case["source"] == "fbm":
        return ctx.fbm_volume(vi, seed)
    if case["source"] == "blob":
        return ctx.blob_volume(vi, case["blobs"], seed, noise=case["noise"])
    if case["source"] == "blob_host":
        return ctx.blob_volume(vi, case["blobs"], seed, noise=case["noise"], placement=lv.BLOB_HOST)
    level = vi.depth - 1
    bricks = _cut(_field(case, seed), vi, level)

    def get_data(node_id, dst, nbytes):
        b = bricks.get(node_id)
        if b is None:
            return False
        ctypes.memmove(dst, b.ctypes.data, nbytes)
        return True

    vol = ctx.callback_volume(vi, get_data)
    vol.load(sorted(bricks))
    return vol


def _table(case, seed):
    if case["tf"] == "default":
        return lv.default_transfer_function()
    return lv.linear_ramp_tf(case["tf_n"]) if case["tf"] == "ramp" else lv.gaussian_peaks_tf(case["tf_n"], seed=seed)


def _camera(case, seed):
    r = np.random.default_rng(seed + 77)
    W, H = case["width"], case["height"]
    if case["camera"] == "inside":
        # along a path through the volume, looking ahead
        eye = np.array([r.uniform(-0.2, 0.2), r.uniform(-0.2, 0.2), 0.45])
        at = eye + np.array([r.uniform(-0.25, 0.25), r.uniform(-0.2, 0.2), -1.0])
        return lv.look_at(eye, at), lv.perspective(60.0, W / H, 0.01, 15.0)
    world = _info(case).world_size
    return lv.orbit_camera(int(r.integers(0, 64)), 64, world, W, H, radius_scale=case["radius"])


def _desc(ctx, case, seed):
    mv, proj = _camera(case, seed)
    lo, hi = VALUES.get(case["dtype"], (0.0, 0.0)) if case["source"] == "field" else (0.0, 0.0)
    return ctx.render_desc(
        mv, proj, case["width"], case["height"], sse=case["sse"], min_lod=case["min_lod"], early_exit=case["early"],
        step_policy=lv.STEP_HALF_VOXEL if case["step"] == "half_voxel" else lv.STEP_REFERENCE,
        filt=lv.FILTER_TRILINEAR if case["filter"] == "trilinear" else lv.FILTER_NEAREST,
        data_range=(lo, hi), synchronous=case["sync"], max_uploads=16)


def _pool_bytes(vi, dtype):
    """A pool that holds the whole octree in the default brick layout."""
    return vi.node_count() * (vi.slot_bytes + 1024) + (64 << 20)


def _views(case, seed):
    """The views of a batch or a burst: (volume case, view case) pairs over three data sets."""
    shapes, r = np.random.default_rng(case["views"]), np.random.default_rng(seed)
    vols = [dict(source="blob", blobs=64, noise=4, voxels="512x512x512", block=64, overlap=1, dtype="u8"),
            dict(source="blob", blobs=64, noise=4, voxels="512x512x512", block=64, overlap=1, dtype="u16"),
            dict(source="fbm", voxels="256x256x256", block=32, overlap=1, dtype="u8")]
    sizes = [(256, 256), (320, 240), (512, 512), (641, 479)]
    if case["sizes"] == "mixed":
        sizes += [(1001, 701), (1280, 720), (1920, 1080)]
    views = []
    for i in range(case["views"]):
        w, h = sizes[int(shapes.integers(0, len(sizes)))]
        views.append((i % 3, dict(vols[i % 3], width=w, height=h, sse=float(r.uniform(0.8, 3.0)), min_lod=0, early=0.99,
                                  step="half_voxel", filter="trilinear", camera="orbit", sync=True,
                                  radius=float(r.uniform(1.3, 2.5)))))
    return vols, views


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    seed = int(seed)
    kind = case["kind"]
    if kind == "select":
        ctx = lv.Context(0, pool_bytes=64 << 20)
        vi = _info(case)
        mv, proj = _camera(case, seed)
        out = torch.empty(min(vi.node_count(), 1 << 17), dtype=torch.int64, device="cuda")
        result = torch.zeros(lv._abi.SELECT_RESULT_WORDS, dtype=torch.int32, device="cuda")
        return dict(kind=kind, ctx=ctx, vi=vi, mv=mv, proj=proj, case=case, out=out, result=result)
    if kind == "histogram":
        vi = _info(case)
        ctx = lv.Context(0, pool_bytes=_pool_bytes(vi, case["dtype"]))
        vol = _volume(ctx, case, seed)
        level = vi.depth - 1
        ids = [int(i) for i in vi.all_nodes() if i.level == level]
        return dict(kind=kind, vol=vol, ctx=ctx, ids=ids, bins=case["bins"], range=VALUES[case["dtype"]])
    if kind in ("batch", "serve"):
        vcases, views = _views(case, seed)
        ctx = lv.Context(0, pool_bytes=3 * GIB)
        vols = [_volume(ctx, v, seed + k) for k, v in enumerate(vcases)]
        tfs = [ctx.transfer_function(lv.gaussian_peaks_tf(256, seed=seed + k)) for k in range(4)]
        items = []
        for i, (k, c) in enumerate(views):
            out = torch.empty((c["height"], c["width"], 4), dtype=torch.float32, device="cuda")
            items.append((vols[k], tfs[i % 4], _desc(ctx, c, seed + i), out))
        for v, t, d, o in items:
            ctx.render(v, t, d, o)
        torch.cuda.synchronize()
        state = dict(kind=kind, items=items, ctx=ctx)
        if kind == "batch":
            state["batch"] = lv.Batch(ctx)
        else:
            state["server"] = lv.Server(ctx)
        return state
    vi = _info(case)
    ctx = lv.Context(0, pool_bytes=min(_pool_bytes(vi, case["dtype"]), 24 * GIB))
    vol = _volume(ctx, case, seed)
    tf = ctx.transfer_function(_table(case, seed))
    desc = _desc(ctx, case, seed)
    out = torch.empty((case["height"], case["width"], 4), dtype=torch.float32, device="cuda")
    if kind == "frame":
        ctx.render(vol, tf, desc, out)  # the view's bricks are resident
        torch.cuda.synchronize()
    return dict(kind=kind, vol=vol, tf=tf, desc=desc, ctx=ctx, out=out)


# -------------------------------------------------------------------- run
def run(state):
    kind, ctx = state["kind"], state["ctx"]
    if kind == "frame":
        return ctx.render(state["vol"], state["tf"], state["desc"], state["out"])
    if kind == "cold":
        ctx.purge()
        return ctx.render(state["vol"], state["tf"], state["desc"], state["out"])
    if kind == "batch":
        state["batch"].render(state["items"])
        return [o for _, _, _, o in state["items"]]
    if kind == "serve":
        tickets = [state["server"].submit(*item) for item in state["items"]]
        for t in tickets:
            state["server"].wait(t)
        return [o for _, _, _, o in state["items"]]
    if kind == "histogram":
        return state["vol"].histogram(state["ids"], state["bins"], state["range"], per_brick=True)
    c = state["case"]
    # on the device, in id order: the selection lists the visible set in no order of its own
    ids, result = ctx.select_visible(state["vi"], state["mv"], state["proj"], c["height"], c["sse"],
                                     out=state["out"].fill_(-1), result=state["result"], sync=False)
    return torch.sort(ids).values, result


# ------------------------------------------------------------------- work
def _samples(case):
    """Samples of a frame without early termination, and the share of the frame's pixels they
    come from: mean ray length inside the volume's box on a coarse grid of pixels, times the
    samples per unit length at the finest level the view can select."""
    vi = _info(case)
    mv, proj = _camera(case, 0)
    o, d, tnp = _rays(mv, proj, 48, 48, np)
    half = np.array(vi.world_size) / 2
    with np.errstate(divide="ignore"):
        a, b = (-half - o) / d, (half - o) / d
    t0, t1 = np.minimum(a, b).max(-1), np.maximum(a, b).min(-1)
    length = np.maximum(t1 - np.maximum(t0, tnp), 0)
    # a voxel projects to at most about `sse` pixels at the near side: coarser levels step wider
    finest = max(_voxels(case)) if case["min_lod"] else min(max(_voxels(case)), 2 * case["height"] / case["sse"])
    n = 2 * finest if case["step"] == "half_voxel" else max(finest, 512)
    return float(length.mean() * n * case["width"] * case["height"])


def _frame_work(case):
    vi = _info(case)
    s = _samples(case)
    voxels = float(np.prod([float(v) for v in _voxels(case)]))
    # a voxel is stepped through once or twice by each of the rays it covers; its side projects
    # to half of `sse` to `sse` pixels where the level is chosen by it
    shared = (2.0 if case["step"] == "half_voxel" else 1.0) * (1.0 if case["min_lod"] else max(1.0, 0.75 * case["sse"]) ** 2)
    read = min(voxels, s / shared) * BYTES[case["dtype"]]
    # the fetched bricks are read at their source and written to the pool first
    stream = 2 * read if case["kind"] == "cold" else 0
    # per sample: 7 interpolations, the position, the table and the blend, about 50 operations
    return {"bytes": 16.0 * case["width"] * case["height"] + read + stream + 16.0 * case["tf_n"] + 8.0 * vi.depth,
            "flops": 50.0 * s}


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        w = [_frame_work(dict(c, kind="frame", tf_n=256)) for _, c in _views(case, 0)[1]]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    if kind in ("frame", "cold"):
        return _frame_work(case)
    vi = _info(case)
    if kind == "histogram":
        L = vi.depth - 1
        voxels = float(np.prod([(vi.root_blocks[a] << L) * vi.block_size[a] for a in range(3)]))
        bricks = voxels / float(np.prod(vi.block_size))
        return {"bytes": voxels * BYTES[case["dtype"]] + 8.0 * case["bins"] * (bricks + 1), "flops": 3.0 * voxels}
    # a visited node is read and its id written: about as many as bricks tile the screen, in depth
    nodes = min(float(vi.node_count()), 16.0 * vi.depth * (1 + case["width"] * case["height"] / (case["block"] * case["sse"]) ** 2))
    return {"bytes": 24.0 * nodes, "flops": 150.0 * nodes}


# ------------------------------------------------------------------ exact
def _rays(mv, proj, W, H, xp):
    """Origin, unit directions (H, W, 3) and the near plane's parameter of every pixel's ray."""
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
    near = p[2, 3] / (p[2, 2] - 1.0)
    tnp = -near / (e[..., 2] / np.linalg.norm(e, axis=-1))
    return eye, d, tnp


def _clamped(i, n):
    return i.clamp(0, n - 1)


def exact(case, seed):
    # volumes made here, one level of detail, in 64 bits; the framework's own generators, whose
    # bytes are theirs, have no value; counts and ids are whole numbers
    if case["kind"] != "frame" or case["source"] != "field":
        return None
    vi = _info(case)
    dev = torch.device("cuda")
    data = _field(case, int(seed))
    W, H, B, L = case["width"], case["height"], vi.block_size, vi.depth - 1
    dims = [vi.root_blocks[a] << L for a in range(3)]
    bm, world = max(dims), [float(np.float32(w)) for w in vi.world_size]
    eye, d, tnp = _rays(*_camera(case, int(seed)), W, H, np)
    eye, d, tnp = (torch.from_numpy(np.ascontiguousarray(x)).to(dev) for x in (eye, d.reshape(-1, 3), tnp.reshape(-1)))
    half = torch.tensor(world, dtype=torch.float64, device=dev) / 2
    a, b = (-half - eye) / d, (half - eye) / d
    tg, thi = torch.minimum(a, b).amax(1), torch.maximum(a, b).amin(1)
    tlo = torch.maximum(tg, tnp)
    hit = torch.nonzero((tg <= thi) & (tlo <= thi)).reshape(-1)
    out = torch.zeros((H * W, 4), dtype=torch.float64, device=dev)
    d, tg, thi, tlo = d[hit], tg[hit], thi[hit], tlo[hit]
    nmax = max(_voxels(case))
    n = 2 * nmax if case["step"] == "half_voxel" else max(nmax, 512)
    k = torch.where(tlo > tg, torch.ceil((tlo - tg) * n), torch.zeros_like(tg))
    tf = torch.from_numpy(_table(case, int(seed)).astype(np.float64)).to(dev)
    lo, hi = VALUES[case["dtype"]]
    flat = data.reshape(-1)
    nz, ny, nx = data.shape
    size = [nx, ny, nz]
    dst = torch.zeros((len(hit), 4), dtype=torch.float64, device=dev)
    rows = torch.arange(len(hit), device=dev)

    def voxel(i):
        # a tap: its position over the whole volume, in the sample's brick where there is no overlap
        return flat[(i[2] * ny + i[1]) * nx + i[0]].double()

    while len(rows):
        t = tg + k / n
        keep = t < thi
        if not bool(keep.all()):
            rows, d, tg, thi, k, t = rows[keep], d[keep], tg[keep], thi[keep], k[keep], t[keep]
            if not len(rows):
                break
        f = [(eye[i] + d[:, i] * t + half[i]) * (bm / world[i]) for i in range(3)]
        cell = [torch.floor(f[i]).clamp_min(0) for i in range(3)]
        cell = [cell[i].clamp_max(dims[i] - 1) if dims[i] == bm else cell[i] for i in range(3)]
        ok = (cell[0] < dims[0]) & (cell[1] < dims[1]) & (cell[2] < dims[2])
        g = [f[i] * B[i] for i in range(3)]
        first = [(cell[i] * B[i]).long() for i in range(3)]
        if case["filter"] == "nearest":
            v = voxel([_clamped(torch.minimum(torch.maximum(torch.floor(g[i]).long(), first[i]), first[i] + B[i] - 1), size[i])
                       for i in range(3)])
        else:
            base = [torch.floor(g[i] - 0.5) for i in range(3)]
            w = [g[i] - 0.5 - base[i] for i in range(3)]
            tap = [[base[i].long(), base[i].long() + 1] for i in range(3)]
            for i in range(3):
                for j in range(2):
                    if min(vi.overlap) == 0:  # every tap stays in the brick
                        tap[i][j] = torch.minimum(torch.maximum(tap[i][j], first[i] - vi.overlap[i]),
                                                  first[i] + B[i] - 1 + vi.overlap[i])
                    tap[i][j] = _clamped(tap[i][j], size[i])
            v = 0
            for z in range(2):
                for y in range(2):
                    for x in range(2):
                        c = voxel([tap[0][x], tap[1][y], tap[2][z]])
                        v = v + c * (w[0] if x else 1 - w[0]) * (w[1] if y else 1 - w[1]) * (w[2] if z else 1 - w[2])
        s = ((v - lo) / (hi - lo) * len(tf) - 0.5).clamp(0, len(tf) - 1)
        i0 = s.floor().long()
        i1 = (i0 + 1).clamp_max(len(tf) - 1)
        q = (s - i0)[:, None]
        src = tf[i0] * (1 - q) + tf[i1] * q
        alpha = 1 - (1 - src[:, 3].clamp_max(255 / 256)) ** (32 / n)
        alpha = torch.where(ok, alpha, torch.zeros_like(alpha))
        cur = dst[rows]
        left = alpha * (1 - cur[:, 3])
        cur = torch.cat([cur[:, :3] + src[:, :3] * left[:, None], (cur[:, 3] + left)[:, None]], 1)
        dst[rows] = cur
        k = k + 1
        go = cur[:, 3] <= case["early"]
        if not bool(go.all()):
            rows, d, tg, thi, k = rows[go], d[go], tg[go], thi[go], k[go]
    out[hit] = dst
    return out.reshape(H, W, 4)
