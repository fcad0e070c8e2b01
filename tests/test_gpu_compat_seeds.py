"""The compat render's noise cells, made on the device from each seed's map: seeds one
after another on one context give what the oracle gives for each (tolerance: that of
the compat parity tests), and the same bits when a seed comes back, on any stream."""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs, workload
from oracle import oracle as O

from test_gpu_compat import assert_close, gpu_volume

pytestmark = pytest.mark.gpu


def test_seeds_in_turn(ctx):
    torch = pytest.importorskip("torch")
    cfg = dict(configs.COMPAT_REF, boards=60)
    wl = workload.build_compat(cfg, width=61, height=37)
    vol = gpu_volume(ctx, wl)
    ov = O.OracleVolume(cfg["dim"], cfg["bounds"], cfg["position"], cfg["mips"])
    ov.set_boards(wl.positions, wl.scales, np.ones(len(wl.scales), np.float32))
    ov.voxelize(wl.sun_direction, *cfg["sun_map"])
    cam = workload.make_camera(wl.cameras[0])
    stream = torch.cuda.Stream()
    first = {}
    for turn, seed in enumerate([1, 0, 77, 0xFFFFFFFF, 77, 1, 12345, 0]):
        sh = cloudgb.CompatShader(noiseSeed=seed, doConeTrace=turn % 2 == 0, numOctaves=3)
        img = sh.coneTrace(vol, cam, stream=stream.cuda_stream if turn % 3 == 0 else None)
        ref = ov.compat_render(cam, sh.params(), wl.sun_direction, O.compat_noise_map(seed))
        assert_close(img, ref, what=str(seed))
        again = sh.coneTrace(vol, cam)
        assert np.array_equal(again, img)
        first.setdefault((seed, turn % 2), img)
        assert np.array_equal(first[seed, turn % 2], img)
    assert np.abs(first[1, 0] - first[77, 0]).max() > 0.01
