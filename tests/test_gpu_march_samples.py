"""The packed list of contributing view samples: region order, the first
`capacity` of them, more than one piece, against the rendered opacity."""
import ctypes

import numpy as np
import pytest

import cloudgb
from cloudgb import _lib, configs
from cloudgb.scene import billboards

pytestmark = pytest.mark.gpu

EYE, TARGET = (0.5, 0.6, -1.2), (0.5, 0.5, 0.5)


def _scene(ctx, boards):
    vol = cloudgb.CloudVolume(64, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, 7, ctx=ctx)
    vol.set_billboards(*billboards(3, boards, ball_radius=0.4, radius_scale=1.2))
    vol.update()
    cloudgb.VoxelizeShader().voxelize(vol, cloudgb.Sun((0.3, 1.0, 0.2), 160, 90))
    return vol


def _march(vol, shader, cam, capacity, room):
    pos = np.full((room, 3), -7.0, np.float32)
    w = np.full(room, -7.0, np.float32)
    n = ctypes.c_int()
    p, c = shader.params(), cam._c()
    _lib.check(_lib.load().cg_march_samples(
        vol.ctx.handle, vol.handle, ctypes.byref(c), ctypes.byref(p),
        pos.ctypes.data_as(_lib.FP), w.ctypes.data_as(_lib.FP), capacity, ctypes.byref(n)),
        "cg_march_samples")
    return pos, w, n.value


def _regions(pos, cam):
    """Each sample's 8 x 4 pixel region in the renderer's order, by projection."""
    lo, hi = (np.float64(b) for b in configs.VOLUME_BOUNDS)
    x = pos.astype(np.float64) / 64 * (hi - lo) + lo + np.array(configs.VOLUME_POSITION) - EYE
    f = np.array(TARGET, np.float64) - EYE
    f /= np.linalg.norm(f)
    s = np.cross(f, (0, 1, 0))
    s /= np.linalg.norm(s)
    u = np.cross(s, f)
    t = np.tan(np.radians(cam.fov_y_degrees) / 2)
    px = ((x @ s) / (x @ f) / (t * cam.width / cam.height) + 1) / 2 * cam.width
    py = (1 - (x @ u) / (x @ f) / t) / 2 * cam.height
    # a sample lies on its pixel's centre ray, half a pixel from the edges
    assert np.abs(px - np.floor(px) - 0.5).max() < 0.25
    px, py = px.astype(int), py.astype(int)
    block = (py // 16) * ((cam.width + 15) // 16) + px // 16
    return block * 8 + (py % 16) // 4 * 2 + (px % 16) // 8


@pytest.mark.parametrize("w,h,boards", [(1, 1, 40), (61, 37, 40), (333, 130, 40), (1600, 900, 60),
                                        (61, 37, 0)])
def test_packed_samples(ctx, w, h, boards):
    vol = _scene(ctx, boards)
    shader = cloudgb.ConeTraceShader(viewSteps=48, vctSteps=8)
    cam = cloudgb.Camera(EYE, TARGET, width=w, height=h)
    _, _, total = _march(vol, shader, cam, 0, 0)
    assert (total > 0) == (boards > 0)
    if w == 1600:
        assert total > (1 << 20)  # more than one piece
    pos, wt, n = _march(vol, shader, cam, total + 9, total + 9)
    assert n == total
    assert (pos[total:] == -7).all() and (wt[total:] == -7).all()
    pos, wt = pos[:total], wt[:total]
    if total:
        assert wt.min() >= 0 and wt.max() <= 1
        assert (np.diff(_regions(pos, cam)) >= 0).all()
    # a pixel's weights sum to its opacity
    alpha = shader.coneTrace(vol, cam)[..., 3].astype(np.float64)
    assert abs(alpha.sum() - wt.astype(np.float64).sum()) <= 1e-5 * alpha.sum() + 1e-9
    for capacity in {1, total // 2, max(total - 1, 0), total}:
        p, q, n = _march(vol, shader, cam, capacity, total + 1)
        assert n == total
        k = min(capacity, total)
        assert np.array_equal(p[:k], pos[:k]) and np.array_equal(q[:k], wt[:k])
        assert (p[k:] == -7).all() and (q[k:] == -7).all()
