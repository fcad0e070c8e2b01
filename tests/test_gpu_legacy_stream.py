"""Calls made while the legacy default stream is busy (a caller's PyTorch work): what
they copied is there for the next call, which does not wait for that stream."""
import ctypes

import numpy as np
import pytest

import cloudgb
from cloudgb import _lib, configs, surrogate
from cloudgb.scene import billboards

pytestmark = pytest.mark.gpu

SUN = cloudgb.Sun((0.3, 1.0, 0.2), 96, 64)
CAM = cloudgb.Camera((0.5, 0.6, -0.9), (0.5, 0.5, 0.5), width=70, height=44)


@pytest.fixture
def busy():
    torch = pytest.importorskip("torch")

    def start():
        torch.cuda.synchronize()
        torch.cuda._sleep(100_000_000)  # half a tenth of a second on the legacy stream
    yield start
    torch.cuda.synchronize()


def _volume(ctx, seed):
    vol = cloudgb.CloudVolume(64, configs.VOLUME_BOUNDS, configs.VOLUME_POSITION, 7, ctx=ctx)
    vol.set_billboards(*billboards(seed, 40, radius_scale=1.5))
    vol.update()
    return vol


def test_a_copy_on_the_device(ctx, busy):
    n = 3000
    net = surrogate.SunMLP(ctx, hidden_layers=2)
    x = np.random.default_rng(1).uniform(0, 1, (n, surrogate.N_FEATURES)).astype(np.float32)
    want = net.infer(x)
    a, b, y = (cloudgb.DeviceBuffer(k) for k in (x.nbytes, x.nbytes, 4 * n))
    a.upload(x)
    b.upload(np.zeros_like(x))
    lib = _lib.load()
    busy()
    _lib.check(lib.cg_memcpy(b.ptr, a.ptr, x.nbytes, 3), "cg_memcpy")
    _lib.check(lib.cg_mlp_infer(net.handle, b.ptr, n, y.ptr, 1, None), "cg_mlp_infer")
    ctx.synchronize()
    assert np.array_equal(y.download((n,)), want)


def test_a_model_and_its_parameters(ctx, busy):
    x = np.random.default_rng(1).uniform(0, 1, (500, surrogate.N_FEATURES)).astype(np.float32)
    old = surrogate.SunMLP(ctx, seed=3, hidden_layers=2)
    want = old.infer(x)
    params = old.get_params()[0]
    busy()
    assert np.array_equal(surrogate.SunMLP(ctx, seed=3, hidden_layers=2).infer(x), want)
    other = surrogate.SunMLP(ctx, seed=4, hidden_layers=2)
    busy()
    other.set_params(params)
    assert np.array_equal(other.infer(x), want)


def test_a_new_volume_and_a_new_frame_graph(ctx, busy):
    shader = cloudgb.ConeTraceShader(viewSteps=32, vctSteps=8, coneLanes=0)
    vol = _volume(ctx, 3)
    cloudgb.VoxelizeShader().voxelize(vol, SUN)
    want = shader.coneTrace(vol, CAM)
    assert want[..., 3].max() > 0.1
    busy()
    fresh = _volume(ctx, 3)
    cloudgb.VoxelizeShader().voxelize(fresh, SUN)
    assert np.array_equal(shader.coneTrace(fresh, CAM), want)
    out = cloudgb.DeviceBuffer(CAM.width * CAM.height * 16)
    out.upload(np.zeros(CAM.width * CAM.height * 4, np.float32))
    busy()
    graph = cloudgb.FrameGraph(ctx, [fresh], SUN, [(fresh, CAM, out)], shader)
    graph.launch()
    ctx.synchronize()
    assert np.array_equal(out.download((CAM.height, CAM.width, 4)), want)
