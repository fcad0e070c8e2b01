"""Device memory of an upload: the bars' list is sized by the bars that the boards
meet, not by boards beside or far outside the volume."""
import numpy as np
import pytest

import cloudgb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _used(torch):
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def _pairs(pos, rad, D, bar):
    """Board-bar pairs of boards in the unit cube's volume of D^3 voxels: the bins that
    hold a voxel centre of each board's box, on the Q20 grid."""
    half, one = 1 << 19, 1 << 20
    q = np.rint(pos.astype(np.float64) * D * one).astype(np.int64)
    rq = np.rint(rad.astype(np.float64) * D * one).astype(np.int64)[:, None]
    lo = np.maximum((q - rq - half + one - 1) // one, 0)
    hi = np.minimum((q + rq - half) // one, D - 1)
    edge = np.array([8, 8, bar])
    n = np.where(lo > hi, 0, hi // edge - lo // edge + 1)
    return int(n.prod(axis=1).sum())


@pytest.mark.parametrize("where", [-0.95, 1.05, 2.6, 40.0])
def test_boards_outside_the_volume_take_no_list(ctx, where):
    """3000 boards of three quarters of the extent beside (-0.95), far outside and
    partly in (1.05) a volume: no more memory than their pairs need."""
    torch = pytest.importorskip("torch")
    vol = cloudgb.CloudVolume(512, (0.0, 1.0), (0.0, 0.0, 0.0), 1,
                              fmt=cloudgb.FORMAT_BF16_FP16, ctx=ctx)
    n = 3000
    pos = np.full((n, 3), 0.5, np.float32)
    pos[:, 0] = where - 0.0001 * np.arange(n) / n
    rad = np.full(n, 0.75, np.float32)
    pos[0], rad[0] = 0.5, 0.05
    pairs = _pairs(pos, rad, 512, 32)
    assert pairs < 2000 or where == 1.05
    before = _used(torch)
    vol.set_billboards(pos, rad)
    vol.update()
    # the records of 3000 boards take a third of a megabyte
    assert _used(torch) - before <= 4 * pairs + (8 << 20)
    vol.close()


def test_a_list_longer_than_the_last(ctx):
    """Boards that move from outside into a volume: the list grows with them."""
    rng = np.random.default_rng(5)
    pos = rng.uniform(-0.5, 0.5, (500, 3)).astype(np.float32)
    rad = rng.choice([0.0, 0.02, 0.2, 0.6], 500).astype(np.float32)
    vol = cloudgb.CloudVolume(72, (-0.5, 0.5), (0.5, 0.5, 0.5), 3, ctx=ctx)
    for shift in (3.0, 1.2, 0.6, 0.0):
        vol.set_billboards(pos + np.float32(shift), rad)
        vol.update()
        cloudgb.VoxelizeShader().voxelize(vol, cloudgb.Sun((0.3, 1.0, 0.2), 24, 16))
        ov = O.OracleVolume(72, (-0.5, 0.5), (0.5, 0.5, 0.5), 3)
        assert ov.set_boards(pos + np.float32(shift), rad, np.ones(500, np.float32), 1.0) == 0
        assert ov.voxelize((0.3, 1.0, 0.2), 24, 16) == 0
        for a, b in zip(vol.read_coverage(), ov.coverage()):
            assert np.array_equal(a, b)
