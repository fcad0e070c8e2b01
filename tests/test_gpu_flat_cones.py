"""Exact sun cones whose first steps lie on one level (walked without clamps from
view samples) against the same cones traced by the whole warp (each step by
itself, clamped): one image with coneLanes 0, one with 32.

Tolerance: the samples are the same, only the order of a cone's sum differs (a
compensated chain, a tree of six FP32 additions): tau moves by at most
6 2^-24 tau, a transmittance by at most max(x e^-x) of that, and the samples'
weights sum to at most 1: 1.4e-7, and as much again for the FP32 blend."""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs
from cloudgb.scene import billboards

pytestmark = pytest.mark.gpu

SUNS = [(0.3, 1.0, 0.2), (-0.7, 0.7, -0.17), (0.05, -1.0, 0.6), (1.0, 0.0, 0.0)]


@pytest.mark.parametrize("dim,mips,fmt", [
    (9, 3, cloudgb.FORMAT_RGBA32F), (33, 5, cloudgb.FORMAT_RGBA32F),
    (100, 7, cloudgb.FORMAT_BF16_FP16), (136, 4, cloudgb.FORMAT_RGBA32F),
    (64, 7, cloudgb.FORMAT_BF16_FP16)])
@pytest.mark.parametrize("cone", [dict(vctSteps=24, vctConeAngle=0.06),
                                  dict(vctSteps=33, vctConeAngle=0.2),
                                  dict(vctSteps=1, vctConeAngle=0.06),
                                  dict(vctSteps=64, vctConeAngle=0.06,
                                       vctConeInitialHeight=0.0)])
def test_flat_steps_read_the_same_samples(ctx, dim, mips, fmt, cone):
    vol = cloudgb.CloudVolume(dim, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, mips, fmt=fmt,
                              ctx=ctx)
    # clouds that reach the faces: samples on them, cones that leave at once
    vol.set_billboards(*billboards(dim, 50, ball_radius=0.6, radius_scale=1.5))
    vol.update()
    for sun in SUNS:
        cloudgb.VoxelizeShader().voxelize(vol, cloudgb.Sun(sun, 96, 64))
        cam = cloudgb.Camera((0.5 + 1.4 * sun[2], 0.7, -1.1), (0.5, 0.5, 0.5), width=45, height=30)
        own = cloudgb.ConeTraceShader(viewSteps=40, coneLanes=0, **cone).coneTrace(vol, cam)
        warp = cloudgb.ConeTraceShader(viewSteps=40, coneLanes=32, **cone).coneTrace(vol, cam)
        assert own[..., 3].max() > 0.1
        assert np.array_equal(own[..., 3], warp[..., 3])
        assert np.abs(own - warp).max() <= 3e-7
