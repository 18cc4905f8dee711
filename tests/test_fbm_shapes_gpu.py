"""The device fBm generator's bytes equal the host generator's for rows that
end within a run and start off a word, one to many octaves, and lacunarities
whose lattice cells change at every voxel or leave the permutation's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block,overlap", [((8, 3, 2), 0), ((7, 9, 5), 1), ((33, 6, 4), 0), ((16, 16, 16), 2),
                                           ((64, 5, 3), 1), ((1, 2, 3), 0)])
@pytest.mark.parametrize("kw", [dict(octaves=1), dict(octaves=6, gain=-0.7, lacunarity=1.7, frequency=3.3),
                                dict(octaves=12, frequency=40.0), dict(octaves=4, lacunarity=-2.5),
                                dict(octaves=16, lacunarity=1e4)])
def test_device_bytes_equal_host(gpu_ctx, block, overlap, kw):
    import livre_gb300 as lv
    for dt in (lv.DT_UINT16, lv.DT_UINT8):
        vi = lv.VolumeInformation([2 * b for b in block], block, overlap, dtype=dt)
        ids = [n.id for n in vi.all_nodes()]
        dev = gpu_ctx.fbm_bricks(vi, ids, 5, **kw).cpu().numpy()
        for k, i in enumerate(ids):
            assert np.array_equal(dev[k], lv.fbm_brick(vi, i, 5, n_threads=4, **kw)), hex(i)
