"""Calls on host rows (features, inference, gradient, cones): repeated calls hold no
more device memory than one, whatever the order of their sizes, and give the
results of the calls on device rows."""
import ctypes

import numpy as np
import pytest

import cloudgb
from cloudgb import _lib, configs, surrogate
from cloudgb.scene import billboards

pytestmark = pytest.mark.gpu


def _used(torch):
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.fixture(scope="module")
def scene(ctx):
    vol = cloudgb.CloudVolume(64, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, 7, ctx=ctx)
    vol.set_billboards(*billboards(3, 40, radius_scale=1.5))
    vol.update()
    cloudgb.VoxelizeShader().voxelize(vol, cloudgb.Sun((0.3, 1.0, 0.2), 64, 64))
    return vol, surrogate.SunMLP(ctx, hidden_layers=2)


def _calls(vol, net, n):
    lib = _lib.load()
    rng = np.random.default_rng(n)
    p = rng.uniform(0.0, 64.0, (n, 3)).astype(np.float32)
    d = (ctypes.c_float * 3)(0.3, 1.0, 0.2)
    f = np.zeros((n, surrogate.N_FEATURES), np.float32)
    _lib.check(lib.cg_mlp_features(vol.handle, net.handle, p.ctypes.data_as(_lib.FP), n, d,
                                   f.ctypes.data_as(_lib.FP), 0, None), "cg_mlp_features")
    y = net.infer(f)
    tau = cloudgb.ConeTraceShader().traceCone(vol, p, (0.3, 1.0, 0.2))
    g = np.zeros(surrogate.N_PARAMS, np.float32)
    loss = ctypes.c_float()
    _lib.check(lib.cg_mlp_gradient(net.handle, f.ctypes.data_as(_lib.FP),
                                   tau.ctypes.data_as(_lib.FP), n, 2.0,
                                   g.ctypes.data_as(_lib.FP), ctypes.byref(loss), 0),
               "cg_mlp_gradient")
    return f, y, tau, g


def test_repeated_calls_hold_no_more_memory(scene):
    torch = pytest.importorskip("torch")
    first = _calls(*scene, 300_000)
    before = _used(torch)
    for _ in range(12):
        again = _calls(*scene, 300_000)
        _calls(*scene, 1000)
    # (one call's rows take 19 MB)
    assert _used(torch) - before <= 4 << 20
    for a, b in zip(first, again):
        assert np.array_equal(a, b)


def test_large_calls_give_their_memory_back(scene):
    torch = pytest.importorskip("torch")
    _calls(*scene, 300_000)
    before = _used(torch)
    _calls(*scene, 3_000_000)
    # 192 MB of rows a call; the gradient's partials (889 MB) stay with the model
    assert _used(torch) - before <= 1100 << 20
    _calls(*scene, 3_000_000)
    assert _used(torch) - before <= 1100 << 20


@pytest.mark.parametrize("n", [1, 127, 5000])
def test_host_rows_equal_device_rows(scene, ctx, n):
    vol, net = scene
    lib = _lib.load()
    f, y, tau, _ = _calls(vol, net, n)
    p = np.random.default_rng(n).uniform(0.0, 64.0, (n, 3)).astype(np.float32)
    d = (ctypes.c_float * 3)(0.3, 1.0, 0.2)
    dp, df, dy = (cloudgb.DeviceBuffer(k * n) for k in (12, 64, 4))
    dp.upload(p)
    _lib.check(lib.cg_mlp_features(vol.handle, net.handle, dp.ptr, n, d, df.ptr, 1, None), "f")
    _lib.check(lib.cg_mlp_infer(net.handle, df.ptr, n, dy.ptr, 1, None), "i")
    ctx.synchronize()
    assert np.array_equal(df.download((n, surrogate.N_FEATURES)), f)
    assert np.array_equal(dy.download((n,)), y)
