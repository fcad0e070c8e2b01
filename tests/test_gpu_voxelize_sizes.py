"""Voxelization over volume sizes whose grids end inside a kernel's unit of work:
brick rows that are not whole warps, blocks of mip children cut by the volume's
face, and levels made by more than one launch."""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs
from cloudgb.scene import billboards
from oracle import oracle as O

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


@pytest.mark.parametrize("dim,mips", [(17, 3), (64, 7), (136, 5), (150, 4), (200, 4)])
def test_coverage_of_touching_and_extreme_balls(ctx, dim, mips):
    """Counts and Q16.16 sums against the oracle, bit for bit, where the splat's
    runs are decided by a hair: centres on voxel centres, faces and quarter
    voxels with radii that put voxel centres on the sphere, balls smaller than
    a voxel and as large as the box, columns touched at their tip, boards
    beyond the faces, and sums that wrap."""
    rng = np.random.default_rng(dim)
    n = 160
    cell = np.float32(1.0 / dim)
    centre = (rng.integers(-2, 4 * dim + 2, (n, 3)) / 4.0).astype(np.float32)  # voxels
    radius = rng.choice([0.0, 0.25, 0.5, 1.0, 1.25, 2.5, 5.0, 6.5, 13.0], n).astype(np.float32)
    # the coverage test keeps 0.9999 of the squared radius: on either side of it
    radius[::3] *= np.float32(1.0 / np.sqrt(0.9999))
    radius[1::7] = rng.uniform(0.2, 0.45 * dim, len(radius[1::7]))
    radius[5], radius[6] = dim, 0.999 * dim
    centre[5:7] = dim / 2 + 0.5
    pos = centre * cell - np.float32(0.5)
    den = rng.choice([0.5, 1.0, 32767.5], n).astype(np.float32)
    vol = cloudgb.CloudVolume(dim, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, mips, ctx=ctx)
    ov = O.OracleVolume(dim, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, mips)
    sun = cloudgb.Sun((0.3, 1.0, 0.2), 40, 24)
    for keep in (slice(0, n), slice(20, 24), slice(0, 0)):  # the bricks of the first scene empty
        p, r, d = pos[keep], radius[keep] * cell, den[keep]
        vol.set_billboards(p, r, d)
        vol.update()
        cloudgb.VoxelizeShader().voxelize(vol, sun)
        assert ov.set_boards(p, r, d) == 0
        assert ov.voxelize(sun.direction, 40, 24) == 0
        cnt, dq = vol.read_coverage()
        ocnt, odq = ov.coverage()
        assert np.array_equal(cnt, ocnt)
        assert np.array_equal(dq, odq)
        raw = vol.read_level(0)
        assert np.array_equal(raw[..., 2], ocnt.astype(np.float32))
        assert np.array_equal(raw[..., 0], odq.astype(np.float32) * np.float32(2.0 ** -16))
        assert np.array_equal(raw[..., 1] > 0, ov.mask() > 0)
