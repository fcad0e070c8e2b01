"""The sun-view map where its tiles' bounds and the sharing of its work decide:
map sizes that cut the tiles, one board to more boards than fill the GPU once,
boards on top of one another, and volumes far from and off the origin."""
import numpy as np
import pytest

import cloudgb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (7, 3), (8, 4), (9, 5), (131, 77), (640, 361)])
@pytest.mark.parametrize("boards", [1, 3, 500, 20000])
def test_map_over_sizes_and_counts(ctx, w, h, boards):
    """Keys (depth and winning board) and positions against the oracle, bit for bit."""
    rng = np.random.default_rng(boards + w)
    dim, mips = 24, 3
    bounds, position = [((-0.5, 0.5), (0.5, 0.5, 0.5)), ((-3.0, 3.0), (40.0, -7.0, 1.0)),
                        ((-0.25, 2.0), (0.0, 0.1, 0.0))][boards % 3]
    size = bounds[1] - bounds[0]
    pos = (rng.uniform(bounds[0] - 0.1 * size, bounds[1] + 0.1 * size, (boards, 3))
           ).astype(np.float32)
    top = 0.6 if boards < 1000 else 0.08
    radius = (size * rng.choice([0.004, 0.02, 0.05, top], boards)).astype(np.float32)
    if boards > 100:  # the same board again: the first of them wins
        pos[50:90] = pos[:40]
        radius[50:90] = radius[:40]
        radius[7] = 0.0
    den = np.ones(boards, np.float32)
    vol = cloudgb.CloudVolume(dim, bounds, position, mips, ctx=ctx)
    ov = O.OracleVolume(dim, bounds, position, mips)
    vol.set_billboards(pos, radius, den)
    vol.update()
    assert ov.set_boards(pos, radius, den) == 0
    for direction in [(0.3, 1.0, 0.2), (-1.0, 0.05, 0.4)]:
        sun = cloudgb.Sun(direction, w, h)
        cloudgb.VoxelizeShader().voxelize(vol, sun)
        assert ov.voxelize(sun.direction, w, h) == 0
        keys, pm = vol.read_sun_map(sun)
        okeys, opm = ov.sun_map()
        assert np.array_equal(keys, okeys)
        assert np.array_equal(pm, opm)
        assert np.array_equal(vol.read_level(0)[..., 1] > 0, ov.mask() > 0)
        cnt, dq = vol.read_coverage()
        assert np.array_equal(cnt, ov.coverage()[0])
