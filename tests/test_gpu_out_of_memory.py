"""Calls that run out of device memory: a volume whose board list or sun map could not
grow holds nothing that was given up on the way, and works again once there is memory."""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs
from cloudgb.scene import billboards
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SUN = cloudgb.Sun((0.3, 1.0, 0.2), 96, 64)


@pytest.fixture
def full():
    """Takes all of the device's memory but half a gigabyte, on demand."""
    torch = pytest.importorskip("torch")
    held = []

    def fill():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        held.append(torch.empty(free - (512 << 20), dtype=torch.uint8, device="cuda"))

    def give_back():
        held.clear()
        torch.cuda.empty_cache()
    yield fill, give_back
    give_back()


def _matches(vol, boards):
    cloudgb.VoxelizeShader().voxelize(vol, SUN)
    ov = O.OracleVolume(vol.dimension, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, 3)
    assert ov.set_boards(*boards, 1.0) == 0
    assert ov.voxelize(SUN.direction, SUN.map_width, SUN.map_height) == 0
    for a, b in zip(vol.read_coverage(), ov.coverage()):
        assert np.array_equal(a, b)


def test_a_board_list_that_cannot_grow(ctx, full):
    fill, give_back = full
    vol = cloudgb.CloudVolume(128, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, 3, ctx=ctx)
    few = billboards(3, 50, radius_scale=1.5)
    vol.set_billboards(*few)
    vol.update()
    _matches(vol, few)
    extent = configs.VOLUME_BOUNDS[1] - configs.VOLUME_BOUNDS[0]
    n = 200_000  # each meets all 4096 bars: a list of 3.3 GB
    many = (np.zeros((n, 3), np.float32), np.full(n, 0.95 * extent, np.float32),
            np.full(n, 0.001, np.float32))
    fill()
    vol.set_billboards(*many)
    with pytest.raises(Exception, match="memory"):
        vol.update()
    # no boards, and none of the old ones' memory
    cloudgb.VoxelizeShader().voxelize(vol, SUN)
    assert vol.activeVoxels() == 0 and vol.info().board_count == 0
    give_back()
    vol.set_billboards(*few)
    vol.update()
    _matches(vol, few)
    vol.close()


def test_a_sun_map_that_cannot_grow(ctx, full):
    fill, give_back = full
    vol = cloudgb.CloudVolume(64, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, 3, ctx=ctx)
    few = billboards(3, 50, radius_scale=1.5)
    vol.set_billboards(*few)
    vol.update()
    _matches(vol, few)
    keys, _ = vol.read_sun_map(SUN)
    fill()
    for side in (6000, 16384):  # 0.3 and 2.1 GB of keys, 0.6 and 4.3 GB of positions
        with pytest.raises(Exception, match="memory"):
            cloudgb.VoxelizeShader().voxelize(vol, cloudgb.Sun(SUN.direction, side, side))
        with pytest.raises(Exception, match="not voxelized"):
            vol.read_sun_map(SUN)
    give_back()
    # the map's old size again
    _matches(vol, few)
    assert np.array_equal(vol.read_sun_map(SUN)[0], keys)
    vol.close()
