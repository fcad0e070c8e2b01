"""New volumes: made without waiting for what is queued on the context, and complete for
the first voxelize, whatever their memory held before and on whichever stream."""
import time

import numpy as np
import pytest

import cloudgb
from cloudgb import configs
from cloudgb.scene import billboards

pytestmark = pytest.mark.gpu

SUN = cloudgb.Sun((0.3, 1.0, 0.2), 96, 64)


def _volume(ctx, dim, mips, fmt, seed):
    vol = cloudgb.CloudVolume(dim, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, mips, fmt=fmt,
                              ctx=ctx)
    vol.set_billboards(*billboards(seed, 40, ball_radius=0.5, radius_scale=1.2))
    vol.update()
    return vol


def _busy(ctx, frames):
    """Queues frames of a millisecond or so each on the context's stream."""
    vol = _volume(ctx, 128, 7, cloudgb.FORMAT_RGBA32F, 1)
    cloudgb.VoxelizeShader().voxelize(vol, SUN)
    cam = cloudgb.Camera((0.5, 0.6, -0.4), (0.5, 0.5, 0.5), width=1920, height=1080)
    out = cloudgb.DeviceBuffer(1920 * 1080 * 16)
    shader = cloudgb.ConeTraceShader(coneLanes=0, numOctaves=3)

    def queue():
        for _ in range(frames):
            shader.coneTrace(vol, cam, out=out)
    queue()
    ctx.synchronize()
    t = time.perf_counter()
    queue()
    ctx.synchronize()
    return queue, time.perf_counter() - t


def test_creation_does_not_wait_for_queued_frames(ctx):
    queue, whole = _busy(ctx, 200)
    for fmt in (cloudgb.FORMAT_RGBA32F, cloudgb.FORMAT_BF16_FP16):
        queue()
        vol = cloudgb.CloudVolume(64, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, 7, fmt=fmt,
                                  ctx=ctx)
        t = time.perf_counter()
        ctx.synchronize()
        left = time.perf_counter() - t
        assert left > 0.4 * whole, (left, whole)
        vol.close()


@pytest.mark.parametrize("fmt", [cloudgb.FORMAT_RGBA32F, cloudgb.FORMAT_BF16_FP16])
@pytest.mark.parametrize("dim,mips", [(64, 7), (33, 5), (136, 4), (8, 1)])
def test_first_voxelize_on_any_stream(ctx, dim, mips, fmt):
    torch = pytest.importorskip("torch")
    shader = cloudgb.ConeTraceShader(viewSteps=40, vctSteps=24)
    cam = cloudgb.Camera((0.5, 0.6, -0.9), (0.5, 0.5, 0.5), width=70, height=44)

    def contents(vol):
        return [vol.read_level(l) for l in range(mips)] + [shader.coneTrace(vol, cam)]
    vol = _volume(ctx, dim, mips, fmt, 5)
    cloudgb.VoxelizeShader().voxelize(vol, SUN)
    want = contents(vol)
    vol.close()
    queue, _ = _busy(ctx, 5)
    streams = [torch.cuda.Stream() for _ in range(2)]
    for turn in range(6):
        # memory that the next volume may get, full of what is neither zero nor a density
        junk = torch.full((int(1.5 * dim ** 3) * 32 // 4 + 1024,), -1e30, device="cuda")
        torch.cuda.synchronize()
        del junk
        torch.cuda.empty_cache()
        if turn % 2:
            queue()
        vol = _volume(ctx, dim, mips, fmt, 5)
        stream = [None, *streams][turn % 3]
        cloudgb.VoxelizeShader().voxelize(
            vol, SUN, stream=stream.cuda_stream if stream else None)
        torch.cuda.synchronize()
        for a, b in zip(contents(vol), want):
            assert np.array_equal(a, b)
        vol.close()
