"""The frame graph's voxelizes run side by side: more and fewer volumes than
branches, a volume listed twice, boards replaced between replays; pixels as the
volumes voxelized and rendered one after another, bit for bit."""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs
from cloudgb.scene import billboards

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [[0], [0, 1, 0], [0, 1, 2, 3, 4, 5, 1, 0], [2, 2, 2, 2, 2, 0]])
def test_frames_equal_the_serial_ones(ctx, order):
    dims = [16, 33, 64, 96, 40, 8]
    sun = cloudgb.Sun((0.3, 1.0, 0.2), 200, 120)
    shader = cloudgb.ConeTraceShader(viewSteps=32, vctSteps=8, coneLanes=0)

    def volumes():
        return [cloudgb.CloudVolume(d, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, 3, ctx=ctx)
                for d in dims]

    def upload(vols, seed):
        for i, v in enumerate(vols):
            v.set_billboards(*billboards(seed + i, 30 + 40 * i))
            v.update()

    vols, serial = volumes(), volumes()
    upload(vols, 5)
    for v in vols:
        cloudgb.VoxelizeShader().voxelize(v, sun)
    cam = cloudgb.Camera((0.5, 0.6, -0.9), (0.5, 0.5, 0.5), width=70, height=44)
    outs = [cloudgb.DeviceBuffer(70 * 44 * 16) for _ in order]
    graph = cloudgb.FrameGraph(ctx, [vols[i] for i in order], sun,
                               [(vols[i], cam, o) for i, o in zip(order, outs)], shader)
    for seed in (5, 50, 90):
        upload(vols, seed)
        upload(serial, seed)
        graph.launch()
        ctx.synchronize()
        for i, o in zip(order, outs):
            cloudgb.VoxelizeShader().voxelize(serial[i], sun)
            want = shader.coneTrace(serial[i], cam)
            assert want[..., 3].max() > 0.1
            assert np.array_equal(o.download((44, 70, 4)), want)
