"""Views in which every sample has lod 0, where the exact renderers take only the
steps in occupied bricks (the single view's with cooperative cones on FP32
volumes, the batch's always), against the renderer that looks at every step
(coneLanes 0): the same samples, so the same opacities bit for bit; and views
with coarser samples, where none skips.

Tolerance of the colours: test_gpu_flat_cones's (the order of a cooperative
cone's sum)."""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs
from cloudgb.scene import billboards

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [cloudgb.FORMAT_RGBA32F, cloudgb.FORMAT_BF16_FP16])
@pytest.mark.parametrize("dim,mips,height", [(8, 3, 40), (33, 5, 121), (64, 7, 210), (64, 7, 30)])
@pytest.mark.parametrize("steps", [1, 7, 48])
def test_steps_in_empty_bricks_change_nothing(ctx, dim, mips, height, steps, fmt):
    vol = cloudgb.CloudVolume(dim, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, mips, fmt=fmt,
                              ctx=ctx)
    # few small boards: most bricks are empty, some rays meet several clouds
    vol.set_billboards(*billboards(dim, 14, ball_radius=0.55, radius_scale=0.8))
    vol.update()
    cloudgb.VoxelizeShader().voxelize(vol, cloudgb.Sun((0.3, 1.0, 0.2), 96, 64))
    kw = dict(viewSteps=steps, vctSteps=8, densityScale=30.0, numOctaves=2)
    for eye in [(0.5, 0.6, -0.9), (1.7, 0.2, 0.7), (0.5, 0.5, 0.5)]:
        target = (0.5, 0.5, 0.5) if eye != (0.5, 0.5, 0.5) else (0.9, 0.6, 0.1)
        cam = cloudgb.Camera(eye, target, width=height + 7, height=height)
        every = cloudgb.ConeTraceShader(coneLanes=0, **kw).coneTrace(vol, cam)
        some = cloudgb.ConeTraceShader(**kw).coneTrace(vol, cam)
        if steps == 48:
            assert every[..., 3].max() > 0.1 and every[..., 3].min() == 0.0 or eye[2] == 0.5
        assert np.array_equal(every[..., 3], some[..., 3])
        assert np.abs(every - some).max() <= 3e-7
        for brick in (4, 8, 16):
            vol.set_occupancy_brick(brick)
            assert np.array_equal(cloudgb.ConeTraceShader(**kw).coneTrace(vol, cam), some)
            out = cloudgb.DeviceBuffer(cam.width * cam.height * 16)
            ctx.render_batch([(vol, cam, out)], cloudgb.ConeTraceShader(**kw), config=(1, 1, brick))
            ctx.synchronize()
            got = out.download((cam.height, cam.width, 4))
            assert np.array_equal(got, every)
        vol.set_occupancy_brick(4)
