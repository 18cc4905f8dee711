"""Histograms over brick shapes and bin counts at the edges of the kernel's
row split, counter copies and voxel-quad reads, against numpy's counts of
the same bytes (exact)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# block (x, y, z), overlap, lv_dtype, numpy type; rows of 64 or more uint8
# voxels are stored as voxel quads
SHAPES = [((64, 64, 64), 1, 1, np.uint8), ((65, 63, 9), 0, 1, np.uint8), ((63, 1, 5), 2, 1, np.uint8),
          ((130, 7, 3), 1, 1, np.uint8), ((30, 31, 33), 1, 1, np.uint8), ((1, 5, 3), 0, 1, np.uint8),
          ((17, 20, 3), 1, 4, np.int8), ((33, 40, 12), 1, 2, np.uint16), ((66, 5, 70), 0, 5, np.int16),
          ((40, 12, 3), 1, 0, np.float32)]


@pytest.mark.parametrize("block,overlap,dtype,ntype", SHAPES)
def test_histogram_shapes(gpu_ctx, block, overlap, dtype, ntype):
    import livre_gb300 as lv
    vi = lv.VolumeInformation([2 * b for b in block], block, overlap, dtype=dtype)
    r = np.random.default_rng(hash((block, dtype)) & 0xFFFF)
    shape = tuple(b + 2 * overlap for b in block[::-1])
    ids = [n.id for n in vi.all_nodes()][:5]
    bricks = {}
    for k, i in enumerate(ids):
        v = r.integers(0, 256, shape) if k % 2 else np.full(shape, 37)  # mixed, and one value
        bricks[i] = np.ascontiguousarray(v.astype(np.uint8).view(np.int8) if ntype == np.int8
                                         else v.astype(ntype))

    def get_data(node_id, dst, nbytes):
        b = bricks[node_id]
        assert b.nbytes == nbytes
        C.memmove(dst, b.ctypes.data, nbytes)
        return True

    vol = gpu_ctx.callback_volume(vi, get_data)
    lo, hi = (-100.0, 120.0) if ntype == np.int8 else (3.0, 250.0)
    for n_bins in (2, 256, 257, 1000, 8192):
        acc, per = vol.histogram(ids, n_bins, (lo, hi), per_brick=True)
        alone = vol.histogram(ids[:1], n_bins, (lo, hi))
        scale_bins = np.float32(n_bins - 1) / (np.float32(hi) - np.float32(lo))
        want = np.zeros((len(ids), n_bins), np.uint64)
        for k, i in enumerate(ids):
            o = overlap
            b = bricks[i][o:shape[0] - o, o:shape[1] - o, o:shape[2] - o].astype(np.float32)
            f = np.floor((b - np.float32(lo)) * scale_bins)
            scale = (2 ** (vi.depth - 1 - (i & 0xF))) ** 3
            want[k] = np.bincount(np.clip(f, 0, n_bins - 1).astype(np.int64).ravel(),
                                  minlength=n_bins).astype(np.uint64) * np.uint64(scale)
        assert (per == want).all(), n_bins
        assert (acc == want.sum(0)).all() and (alone == want[0]).all(), n_bins
    vol.close()
