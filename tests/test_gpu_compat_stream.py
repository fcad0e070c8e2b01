"""Compat renders on a caller's stream with a device image return while the GPU still
blends the boards: a render sees the list uploaded before it and not the one
uploaded right after it, whether the records keep their places or move."""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs, workload

pytestmark = pytest.mark.gpu


def _scene(ctx):
    cfg = configs.COMPAT_REF
    wl = workload.build_compat(cfg, boards=400, width=1280, height=720)
    vol = cloudgb.CloudVolume(cfg["dim"], cfg["bounds"], cfg["position"], cfg["mips"], ctx=ctx)
    return wl, vol, workload.make_camera(wl.cameras[0])


def _upload(vol, wl, lst):
    seed, n = lst
    pick = np.random.default_rng(seed).permutation(len(wl.scales))[:n]
    vol.set_billboards(wl.positions[pick], wl.scales[pick])
    vol.update()


@pytest.mark.parametrize("counts", [(200, 200, 200, 200), (200, 120, 200, 1), (10, 100, 400, 0)])
def test_uploads_right_behind_renders(ctx, counts):
    torch = pytest.importorskip("torch")
    wl, vol, cam = _scene(ctx)
    shader = cloudgb.CompatShader(doConeTrace=False)
    lists = [(7 + i, n) for i, n in enumerate(counts)]
    outs = [cloudgb.DeviceBuffer(cam.width * cam.height * 16) for _ in lists]
    streams = [torch.cuda.Stream() for _ in range(2)]
    _upload(vol, wl, (1, 400 if counts[0] != 10 else 5))
    shader.coneTrace(vol, cam, out=outs[0], stream=streams[0].cuda_stream)
    for i, (lst, out) in enumerate(zip(lists, outs)):
        _upload(vol, wl, lst)
        # (a context's renders share its lists: on two streams they follow each other)
        streams[i % 2].wait_stream(streams[1 - i % 2])
        shader.coneTrace(vol, cam, out=out, stream=streams[i % 2].cuda_stream)
    _upload(vol, wl, (1, 400))
    torch.cuda.synchronize()
    _, other, _ = _scene(ctx)
    for lst, out in zip(lists, outs):
        _upload(other, wl, lst)
        want = shader.coneTrace(other, cam)
        got = out.download((cam.height, cam.width, 4))
        assert np.array_equal(got, want)
        if lst[1] >= 100:
            assert want.std() > 0.05


def test_host_image_behind_an_upload(ctx):
    """A host image is complete when the call returns, on a caller's stream too."""
    torch = pytest.importorskip("torch")
    wl, vol, cam = _scene(ctx)
    shader = cloudgb.CompatShader(doConeTrace=False)
    stream = torch.cuda.Stream()
    for lst in [(3, 400), (4, 150), (5, 399)]:
        _upload(vol, wl, lst)
        got = shader.coneTrace(vol, cam, stream=stream.cuda_stream)
        assert np.array_equal(got, shader.coneTrace(vol, cam))
