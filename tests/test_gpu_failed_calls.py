"""A call that failed is not reported again by the next one."""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs
from cloudgb.scene import billboards

pytestmark = pytest.mark.gpu


def test_a_failed_allocation_is_reported_once(ctx):
    vol = cloudgb.CloudVolume(64, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, 7, ctx=ctx)
    vol.set_billboards(*billboards(3, 40, radius_scale=1.5))
    vol.update()
    sun = cloudgb.Sun((0.3, 1.0, 0.2), 64, 64)
    cam = cloudgb.Camera((0.5, 0.6, -0.9), (0.5, 0.5, 0.5), width=70, height=44)
    cloudgb.VoxelizeShader().voxelize(vol, sun)
    want = cloudgb.ConeTraceShader().coneTrace(vol, cam)
    for again in (lambda: vol.update(),
                  lambda: cloudgb.VoxelizeShader().voxelize(vol, sun),
                  lambda: cloudgb.ConeTraceShader().coneTrace(vol, cam),
                  lambda: cloudgb.CompatShader(doConeTrace=False).coneTrace(vol, cam)):
        with pytest.raises(Exception, match="memory"):
            cloudgb.DeviceBuffer(1 << 44)  # more than any device has
        again()
        vol.update()
        cloudgb.VoxelizeShader().voxelize(vol, sun)
    assert np.array_equal(cloudgb.ConeTraceShader().coneTrace(vol, cam), want)
