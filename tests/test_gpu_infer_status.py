"""Inference and the status words: an inference clears nothing that another call has
recorded or still counts in, whenever the GPU gets to it."""
import ctypes

import numpy as np
import pytest

import cloudgb
from cloudgb import _lib, configs, surrogate
from cloudgb.scene import billboards

pytestmark = pytest.mark.gpu


def _render(ctx, net):
    vol = cloudgb.CloudVolume(64, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, 7, ctx=ctx)
    vol.set_billboards(*billboards(3, 40, ball_radius=0.4, radius_scale=1.2))
    vol.update()
    cloudgb.VoxelizeShader().voxelize(vol, cloudgb.Sun((0.3, 1.0, 0.2), 160, 90))
    shader = cloudgb.ConeTraceShader(useMlp=True, mlp=net, viewSteps=48)
    cam = cloudgb.Camera((0.5, 0.6, -1.2), (0.5, 0.5, 0.5), width=160, height=90)
    return lambda: shader.coneTrace(vol, cam)


def _net(ctx):
    net = surrogate.SunMLP(ctx, hidden_layers=2)
    cfg = _lib.cg_mlp_config()
    _lib.check(_lib.load().cg_mlp_get_config(net.handle, ctypes.byref(cfg)))
    cfg.dimension = 64
    cfg.feature_max[:] = [0.05] * 16  # most samples lie outside: the exact cone's
    _lib.check(_lib.load().cg_mlp_configure(net.handle, ctypes.byref(cfg)))
    return net


def test_an_inference_behind_a_render_leaves_its_counts(ctx):
    torch = pytest.importorskip("torch")
    net = _net(ctx)
    render = _render(ctx, net)
    net.infer(np.zeros((1, surrogate.N_FEATURES), np.float32))  # (loads its kernel)
    render()
    want = ctx.last_samples(), ctx.mlp_fallbacks()
    assert want[0] > 1000 and want[1] > 100
    n = 5000
    x = torch.rand((n, surrogate.N_FEATURES), device="cuda")
    y = torch.full((n,), -7.0, device="cuda")
    late = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(late):
        torch.cuda._sleep(200_000_000)  # a tenth of a second
    _lib.check(_lib.load().cg_mlp_infer(net.handle, ctypes.c_void_p(x.data_ptr()), n,
                                        ctypes.c_void_p(y.data_ptr()), 1,
                                        ctypes.c_void_p(late.cuda_stream)), "cg_mlp_infer")
    image = render()
    assert not late.query()  # (the inference has not run yet)
    assert (ctx.last_samples(), ctx.mlp_fallbacks()) == want
    assert np.array_equal(y.cpu().numpy(), net.infer(x.cpu().numpy()))
    # after an inference there is no render to speak of, after a render there is
    assert (ctx.last_samples(), ctx.mlp_fallbacks()) == (0, 0)
    assert np.array_equal(render(), image)
    assert (ctx.last_samples(), ctx.mlp_fallbacks()) == want


def test_a_recorded_timeout_is_not_an_inference_s(ctx):
    """A wait probe's fault is its own: an inference after it succeeds."""
    lib = _lib.load()
    net = surrogate.SunMLP(ctx, hidden_layers=1)
    x = np.random.default_rng(1).uniform(0, 1, (300, surrogate.N_FEATURES)).astype(np.float32)
    before = net.infer(x)
    waited = ctypes.c_uint64()
    assert lib.cg_context_check_wait_timeout(ctx.handle, 1000, ctypes.byref(waited)) == 6
    fb = ctypes.c_uint64()
    assert lib.cg_context_mlp_fallbacks(ctx.handle, ctypes.byref(fb)) == 6
    assert np.array_equal(net.infer(x), before)
    assert ctx.mlp_fallbacks() == 0
