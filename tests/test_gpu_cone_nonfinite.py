"""The reference's weighted cone at positions that are not finite: a NaN or an
infinity gives a NaN, whatever the other coordinates, and changes nothing else."""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs
from cloudgb.scene import billboards

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [cloudgb.FORMAT_RGBA32F, cloudgb.FORMAT_BF16_FP16])
@pytest.mark.parametrize("dim,mips", [(16, 1), (33, 5), (64, 7)])
def test_reference_cone_of_positions_not_finite(ctx, dim, mips, fmt):
    vol = cloudgb.CloudVolume(dim, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, mips, fmt=fmt,
                              ctx=ctx)
    vol.set_billboards(*billboards(3, 40, radius_scale=1.5))
    vol.update()
    sun = cloudgb.Sun((0.3, 1.0, 0.2), 64, 64)
    cloudgb.VoxelizeShader().voxelize(vol, sun)
    shader = cloudgb.ConeTraceShader(coneMode=1, vctSteps=9, vctConeAngle=0.4)
    rng = np.random.default_rng(dim)
    p = rng.uniform(-3.0, dim + 3.0, (96, 3)).astype(np.float32)
    p[60] = 3e38, 3e38, 3e38  # finite, though their sum is not
    p[61] = -3e38, 0.5, 3e38
    base = shader.traceCone(vol, p, sun.direction)
    assert np.isfinite(base).all() and base.max() > 0
    q = p.copy()
    odd = []
    for a in range(3):
        for k, value in enumerate((np.nan, np.inf, -np.inf)):
            odd.append(20 + 3 * a + k)
            q[odd[-1], a] = value
    q[40] = np.inf, -np.inf, np.nan
    q[41] = np.nan
    odd += [40, 41]
    got = shader.traceCone(vol, q, sun.direction)
    assert np.isnan(got[odd]).all()
    rest = np.setdiff1d(np.arange(len(p)), odd)
    assert np.array_equal(got[rest], base[rest])
