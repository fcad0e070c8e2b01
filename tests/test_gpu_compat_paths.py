"""The compat render's size rules against the oracle: tile lists ordered by rank,
in shared memory and in place, octaves made in pairs and alone, noise
coordinates too large for the short floor, and levels of one texel.

Tolerance: that of the compat parity tests (1e-4 but for 0.05 % of the values,
1e-3 for all).  An octave of weight 1e-7 at a frequency that takes the general
path moves a value by at most 8 steps x 4 opacity x 1e-7 / 7 < 1e-6.
"""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs, workload
from oracle import oracle as O

from test_gpu_compat import assert_close, gpu_volume

pytestmark = pytest.mark.gpu


def _scene(ctx, boards, w, h, back=1.0):
    cfg = dict(configs.COMPAT_REF, boards=boards)
    wl = workload.build_compat(cfg, width=w, height=h)
    vol = gpu_volume(ctx, wl)
    ov = O.OracleVolume(cfg["dim"], cfg["bounds"], cfg["position"], cfg["mips"])
    ov.set_boards(wl.positions, wl.scales, np.ones(len(wl.scales), np.float32))
    ov.voxelize(wl.sun_direction, *cfg["sun_map"])
    c = dict(wl.cameras[0])
    c["eye"] = tuple(np.array(c["target"]) + back * (np.array(c["eye"]) - c["target"]))
    return wl, vol, ov, workload.make_camera(c)


@pytest.mark.parametrize("boards", [1, 127, 128, 129, 700, 4096, 4097])
def test_list_lengths(ctx, boards):
    """One tile in which nearly every board has an entry."""
    wl, vol, ov, cam = _scene(ctx, boards, 8, 8, back=3.0)
    sh = cloudgb.CompatShader(transmittanceCutoff=0.0, doNoiseSample=False)
    ref = ov.compat_render(cam, sh.params(), wl.sun_direction, O.compat_noise_map(1))
    assert_close(sh.coneTrace(vol, cam), ref, what=str(boards))


@pytest.mark.parametrize("octaves", [0, 1, 2, 3, 5])
def test_octaves(ctx, octaves):
    wl, vol, ov, cam = _scene(ctx, 40, 61, 37)
    sh = cloudgb.CompatShader(numOctaves=octaves, doConeTrace=octaves == 2, freqStep=2.0)
    ref = ov.compat_render(cam, sh.params(), wl.sun_direction, O.compat_noise_map(1))
    img = sh.coneTrace(vol, cam)
    assert_close(img, ref, what=str(octaves))


def test_large_noise_coordinates(ctx):
    wl, vol, ov, cam = _scene(ctx, 40, 61, 37)
    one = cloudgb.CompatShader(numOctaves=1).coneTrace(vol, cam)
    far = cloudgb.CompatShader(numOctaves=2, freqStep=1e7, persStep=1e-7).coneTrace(vol, cam)
    assert np.abs(one - far).max() <= 1e-6 * 40  # 40 boards at most over a pixel
    assert one.std() > 0.01
