"""The exact sun cone over the density quads (two wide loads per trilinear
sample) against the FP64 oracle on the same stored levels: level sizes that are
not multiples of the brick, both storage formats, schedules that stay in one
level, cross several or start below the first level with quads, cones along
every diagonal sense and an axis, and positions on, near and outside the faces.

Tolerance, from the arithmetic: a sample's coordinate is rounded to FP32 within
D 2^-23 voxels, and a trilinear sample changes by at most Rmax / texel per
voxel on each axis (texel >= 4 voxels where quads are used, >= 1 below); the
weights of a cone sum to its length in world units, at most sqrt(3) plus the
widened faces; the sum itself is compensated (1e-6 relative)."""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs
from cloudgb.scene import billboards
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(33, 5, cloudgb.FORMAT_RGBA32F), (100, 7, cloudgb.FORMAT_BF16_FP16),
          (64, 7, cloudgb.FORMAT_BF16_FP16), (136, 3, cloudgb.FORMAT_RGBA32F),
          (64, 2, cloudgb.FORMAT_RGBA32F)]
SUNS = [(0.3, 1.0, 0.2), (-0.7, 0.7, -0.17), (0.05, -1.0, 0.6), (1.0, 0.0, 0.0)]
CONES = [dict(vctSteps=24, vctConeAngle=0.06), dict(vctSteps=33, vctConeAngle=0.4),
         dict(vctSteps=64, vctConeAngle=0.2, vctLodOffset=1.25),
         dict(vctSteps=16, vctConeAngle=0.1, vctConeMinRadius=0.4), dict(vctSteps=1)]


def _positions(rng, D):
    p = rng.uniform(-6.0, D + 6.0, (160, 3))
    p[:40] = rng.uniform(0.2 * D, 0.8 * D, (40, 3))
    for a in range(3):
        p[40 + 10 * a:50 + 10 * a, a] = 0.0
        p[70 + 10 * a:80 + 10 * a, a] = D
    p[100:120] = np.round(p[100:120])
    return p.astype(np.float32)


@pytest.mark.parametrize("dim,mips,fmt", SHAPES)
def test_cones_over_quads_match_oracle(ctx, dim, mips, fmt):
    rng = np.random.default_rng(dim)
    pos, rad, den = billboards(dim, 60, radius_scale=1.5)
    vol = cloudgb.CloudVolume(dim, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, mips, fmt=fmt,
                              ctx=ctx)
    vol.set_billboards(pos, rad, den)
    vol.update()
    cloudgb.VoxelizeShader().voxelize(vol, cloudgb.Sun(SUNS[0], 64, 64))
    levels = []
    for l in range(mips):
        raw = vol.read_level(l)
        if fmt == cloudgb.FORMAT_BF16_FP16:
            out = np.zeros(raw.shape + (4,), np.float64)
            out[..., 0] = (raw << 16).view(np.float32)
            out[..., 1] = (raw >> 16).astype(np.uint16).view(np.float16)
            raw = out
        levels.append(raw.astype(np.float64))
    ov = O.OracleVolume(dim, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, mips)
    ov.set_pyramid(levels)
    rmax = float(levels[0][..., 0].max())
    assert rmax > 0
    pts = _positions(rng, dim)
    for cone in CONES:
        shader = cloudgb.ConeTraceShader(**dict(dict(vctConeMinRadius=2.0), **cone))
        texel = 1.0 if shader.vctConeMinRadius < 2.0 or mips < 3 else 4.0
        atol = 3.0 * dim * 2.0 ** -23 * rmax / texel * 2.0
        for s in SUNS:
            sun = cloudgb.Sun(s)
            got = shader.traceCone(vol, pts, sun.direction).astype(np.float64)
            ref = ov.trace_cones(pts.astype(np.float64), sun.direction,
                                 O.params_from_shader(shader))
            np.testing.assert_allclose(got, ref, rtol=1e-6, atol=atol, err_msg=f"{cone} {s}")
            if shader.vctSteps > 1:
                assert ref.max() > 0


def test_cone_of_a_nan_or_distant_position(ctx):
    """Positions no sample can come from: outside the widened box 0, and a NaN
    neither faults nor changes its neighbours."""
    vol = cloudgb.CloudVolume(64, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, 7, ctx=ctx)
    vol.set_billboards(*billboards(3, 40, radius_scale=1.5))
    vol.update()
    sun = cloudgb.Sun((0.3, 1.0, 0.2), 64, 64)
    cloudgb.VoxelizeShader().voxelize(vol, sun)
    shader = cloudgb.ConeTraceShader()
    p = np.full((64, 3), 30.0, np.float32)
    base = shader.traceCone(vol, p, sun.direction)
    assert base[0] > 0 and (base == base[0]).all()
    p[1] = np.nan
    p[2] = np.inf
    p[3] = -np.inf
    p[4] = 1e30
    p[5] = (30.0, -3e38, 30.0)
    p[6] = (-1e9, 30.0, 30.0)
    got = shader.traceCone(vol, p, sun.direction)
    assert (got[2:7] == 0).all()
    assert (got[7:] == base[7:]).all() and got[0] == base[0]
