"""Voxelization over volume sizes whose grids end inside a kernel's unit of work:
brick rows that are not whole warps, blocks of mip children cut by the volume's
face, and levels made by more than one launch."""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs
from cloudgb.scene import billboards

pytestmark = pytest.mark.gpu


def _volume(ctx, dim, mips, fmt, boards=40, seed=0):
    vol = cloudgb.CloudVolume(dim, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, mips, fmt=fmt,
                              ctx=ctx)
    # some boards reach the faces of the volume
    vol.set_billboards(*billboards(dim + seed, boards, ball_radius=0.5, radius_scale=1.2))
    vol.update()
    cloudgb.VoxelizeShader().voxelize(vol, cloudgb.Sun((0.3, 1.0, 0.2), 160, 90))
    return vol


def _unpack(raw, fmt):
    if fmt == cloudgb.FORMAT_RGBA32F:
        return raw
    return np.stack([(raw << 16).view(np.float32),
                     (raw >> 16).astype(np.uint16).view(np.float16).astype(np.float32)], axis=-1)


@pytest.mark.parametrize("dim,mips", [(16, 5), (33, 6), (100, 7), (140, 8), (264, 9)])
@pytest.mark.parametrize("fmt", [cloudgb.FORMAT_RGBA32F, cloudgb.FORMAT_BF16_FP16])
def test_coarse_levels_are_the_means_of_the_finer_ones(ctx, dim, mips, fmt):
    """Every level above those the splat makes is the fixed-order mean of the
    stored finer level, in FP32 and rounded once: bit for bit."""
    vol = _volume(ctx, dim, mips, fmt)
    first = 3 if dim % 8 == 0 else 0
    fine = _unpack(vol.read_level(first), fmt)
    for l in range(first, mips - 1):
        n = max(1, dim >> (l + 1))
        c = fine[:2 * n, :2 * n, :2 * n]

        def at(a, b, k):
            return c[k::2, b::2, a::2]

        m = ((((at(0, 0, 0) + at(1, 0, 0)) + (at(0, 1, 0) + at(1, 1, 0))) +
              ((at(0, 0, 1) + at(1, 0, 1)) + (at(0, 1, 1) + at(1, 1, 1)))) * np.float32(0.125))
        raw = vol.read_level(l + 1)
        if fmt == cloudgb.FORMAT_RGBA32F:
            assert np.array_equal(raw, m), l
        else:
            bits = np.ascontiguousarray(m[..., 0]).view(np.uint32)
            r = (bits + 0x7FFF + ((bits >> 16) & 1)) >> 16  # round to nearest even
            assert np.array_equal(raw & 0xFFFF, r), l
            assert np.array_equal((raw >> 16).astype(np.uint16).view(np.float16),
                                  m[..., 1].astype(np.float16)), l
        fine = _unpack(raw, fmt)
    assert fine[..., 0].max() > 0


@pytest.mark.parametrize("dim,mips", [(8, 3), (33, 5), (100, 7), (140, 3), (264, 9)])
def test_images_do_not_depend_on_the_brick(ctx, dim, mips):
    """The default bricks' dilation against the wider ones': an unoccupied
    brick reads 0, so the same pixels come out, whichever way the rays go."""
    vol = _volume(ctx, dim, mips, cloudgb.FORMAT_RGBA32F, seed=1)
    shader = cloudgb.ConeTraceShader(viewSteps=48, vctSteps=8)
    for eye in [(0.5, 0.6, -1.2), (1.9, 0.2, 0.7), (0.3, -0.9, 1.4)]:
        cam = cloudgb.Camera(eye, (0.5, 0.5, 0.5), width=61, height=37)
        images = []
        for brick in (4, 8, 16, 4):
            vol.set_occupancy_brick(brick)
            images.append(shader.coneTrace(vol, cam).copy())
        assert images[0][..., 3].max() > 0.1
        for im in images[1:]:
            assert np.array_equal(im, images[0])
