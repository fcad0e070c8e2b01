"""The work that a program has this library do, as cases that can be timed and
checked: single calls and whole frames over the sizes of the repository's own
workloads (cloudgb/configs.py), and draws from the ranges around them.

kinds, and what each stands for in use
  frame     one frame of an animation: the boards are uploaded, the volume is
            voxelized and one view is rendered into a device image, with the
            exact sun cone (layers = 0) or the learned surrogate (layers > 0)
  render    another view of a volume that stands still
  voxelize  moved boards voxelized, then the sun's optical depth asked at
            positions of interest (the cloud's shadow on other objects)
  cones     exact sun cones at many device-resident positions (labels)
  batch     many clouds and views as one frame graph, boards uploaded before
  compat    the reference's own image formation, one view
  samples   a training view: the renderer's first n samples, their labels and
            their features, on the host as the training-set builder keeps them
  infer     the network alone over device-resident feature rows
  gradient  loss and gradient of one set of rows
  train     a run of optimiser steps over device-resident rows
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cloud-renderer_gb300"))
import cloudgb  # noqa: E402
from cloudgb import _lib, surrogate  # noqa: E402

SUN = (0.3, 1.0, 0.2)
SUN_MAP = (1280, 720)
CENTRE = (0.5, 0.5, 0.5)   # the unit cube: centre +- 0.5
BALL = 0.35                # board centres lie in a ball of this radius
RADII = (0.05, 0.15)       # times the case's radius scale
EYE_DISTANCE = 1.5
MIN_RADIUS = 2.0           # floor of the sun cone's radius, level-0 voxels
CONE_H0 = 1.0
AMBIENT = 0.3
NOISE = dict(seed=7, freq=4.0, lac=2.0, gain=0.5)
CUTOFF = 1e-5
NIN, NH, NPARAM = 16, 64, 9473
TAU_SCALE = 1.0
SIGMA = 2.0                # extinction of the training loss

# the compat scene: the reference's own scale (a 32^3 volume of bounds +-5)
COMPAT_POS = (25.0, 0.0, 0.0)
COMPAT_SUN = (-20.0, 20.0, -5.0)
COMPAT_MAP = (256, 256)


def _scene(dim, mips, fmt, boards, rscale, sigma):
    return dict(dim=dim, mips=mips, fmt=fmt, boards=boards, rscale=rscale, sigma=sigma)


def _view(w, h, steps, sun_steps, half, octaves):
    return dict(width=w, height=h, view_steps=steps, sun_steps=sun_steps, half=half,
                octaves=octaves)


SMALL = _scene(64, 7, "rgba32f", 64, 1.0, 8.0)
MEDIUM = _scene(256, 8, "rgba32f", 4096, 0.5, 2.0)
MEDIUM16 = dict(MEDIUM, fmt="bf16")
LARGE16 = _scene(512, 9, "bf16", 16384, 0.5, 2.0)
VIEW_1080P = _view(1920, 1080, 64, 24, 0.03, 4)


def listed():
    return [
        # the smallest frame: launches and latency count
        dict(name="frame_64cube_256px", kind="frame", layers=0, **SMALL,
             **_view(256, 256, 32, 16, 0.05, 0)),
        # the headline frame: half-precision volume and the named three-layer network
        dict(name="frame_256cube_1080p_mlp3", kind="frame", layers=3, **MEDIUM16, **VIEW_1080P),
        # the exact renderer at the same size, FP32
        dict(name="render_256cube_1080p", kind="render", layers=0, **MEDIUM, **VIEW_1080P),
        # the largest view: 4K over 512^3, the exact cone on the half-precision volume
        dict(name="render_512cube_4k_bf16", kind="render", layers=0, **LARGE16,
             **_view(3840, 2160, 128, 32, 0.03, 5)),
        # voxelization alone, ordinary and largest
        dict(name="voxelize_256cube", kind="voxelize", n=4096, sun_steps=24, half=0.03, **MEDIUM),
        dict(name="voxelize_512cube_bf16", kind="voxelize", n=4096, sun_steps=32, half=0.03,
             **LARGE16),
        # labels of a training scene
        dict(name="cones_250k", kind="cones", n=250000, sun_steps=24, half=0.03, **MEDIUM16),
        # uneven clouds and views in one launch
        dict(name="batch_12clouds_32views", kind="batch", clouds=12, views=32, max_dim=256,
             max_boards=4096, max_pixels=1920 * 1080, scene=17),
        # the reference's look at its own scale
        dict(name="compat_1080p", kind="compat", boards=200, width=1920, height=1080, dim=32,
             mips=4),
        # a view of the training set: its share of four million samples
        dict(name="samples_480x270", kind="samples", n=62500, **MEDIUM16,
             **_view(480, 270, 64, 24, 0.03, 4)),
        # the network on a ragged number of rows
        dict(name="infer_200001_mlp2", kind="infer", layers=2, n=200001),
        # one hundred steps at the named batch
        dict(name="train_16384x100_mlp3", kind="train", layers=3, n=400000, batch=16384,
             steps=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "render", "render", "voxelize", "cones", "batch",
                       "compat", "samples", "infer", "gradient", "train"])
    if kind == "infer":
        return dict(kind=kind, layers=rng.randint(1, 3), n=_log(rng, 1, 2000000))
    if kind == "gradient":
        return dict(kind=kind, layers=rng.randint(1, 3), n=_log(rng, 100, 100000))
    if kind == "train":
        return dict(kind=kind, layers=rng.randint(1, 3), n=_log(rng, 5000, 400000),
                    batch=128 * _log(rng, 1, 128), steps=rng.randint(1, 100))
    if kind == "compat":
        w = _log(rng, 128, 1920)
        return dict(kind=kind, boards=_log(rng, 20, 200), width=w,
                    height=max(16, int(w * rng.uniform(0.5, 0.75))), dim=rng.choice([32, 32, 48]),
                    mips=4)
    if kind == "batch":
        return dict(kind=kind, clouds=rng.randint(2, 12), views=rng.randint(3, 32),
                    max_dim=rng.choice([96, 192, 256]), max_boards=_log(rng, 512, 4096),
                    max_pixels=_log(rng, 16384, 1000000), scene=rng.randint(1, 1 << 20))
    dim = rng.choice([32, 48, 64, 96, 100, 128, 160, 192, 250, 256, 256, 320, 384])
    full = int(math.log2(dim)) + 1
    scene = _scene(dim, max(4, full - rng.randint(0, 1)), rng.choice(["rgba32f", "bf16"]),
                   _log(rng, 16, 8192), round(rng.uniform(0.4, 1.0), 3), rng.choice([2.0, 8.0]))
    cone = dict(sun_steps=rng.choice([16, 20, 24, 32]), half=rng.choice([0.03, 0.05, 0.1]))
    if kind == "voxelize":
        return dict(kind=kind, n=_log(rng, 1, 20000), **cone, **scene)
    if kind == "cones":
        return dict(kind=kind, n=_log(rng, 1, 500000), **cone, **scene)
    if kind == "samples":
        w = _log(rng, 64, 480)
        return dict(kind=kind, n=_log(rng, 500, 62500), width=w, height=max(16, int(w * 0.5625)),
                    view_steps=64, octaves=4, **cone, **dict(scene, fmt="bf16"))
    w = _log(rng, 96, 1920)
    view = dict(width=w, height=max(32, int(w * rng.uniform(0.5, 1.0))),
                view_steps=rng.choice([32, 48, 64, 96]), octaves=rng.randint(0, 5))
    return dict(kind=kind, layers=rng.choice([0, 0, 2, 3]) if kind == "frame" else 0, **scene,
                **cone, **view)


# ---- inputs ------------------------------------------------------------------


def _rng(case, seed, salt=0):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, int(seed) >> 31, salt,
                                  int(case.get("boards", 0))])


def _boards(rng, n, rscale):
    """Offsets from the volume's centre, radii and densities."""
    d = rng.normal(size=(n, 3))
    d *= (BALL * rng.random(n) ** (1 / 3) / np.linalg.norm(d, axis=1))[:, None]
    r = rng.uniform(*RADII, n) * rscale
    return d.astype(np.float32), r.astype(np.float32), rng.uniform(0.5, 1.0, n).astype(np.float32)


def _eye(rng):
    while True:
        d = rng.normal(size=3)
        d /= np.linalg.norm(d)
        if abs(d[1]) < 0.95:
            return tuple(float(c + EYE_DISTANCE * x) for c, x in zip(CENTRE, d))


def _camera(rng, w, h):
    return dict(eye=_eye(rng), target=CENTRE, fov=60.0, width=w, height=h)


def _probes(rng, n, dim):
    """Positions in level-0 voxels, in and around the cloud, near the sun's
    far side too."""
    return (rng.uniform(0.05, 0.95, (n, 3)) * dim).astype(np.float32)


def _net_params(layers, rng):
    """He-uniform weights and small biases in the library's flat layout."""
    p = np.zeros(NPARAM, np.float32)

    def fill(at, count, bound):
        p[at:at + count] = rng.uniform(-bound, bound, count)

    fill(0, 1024, math.sqrt(6 / 16))
    fill(1024, 64, 0.1)
    if layers >= 2:
        fill(1088, 4096, math.sqrt(6 / 64))
        fill(5184, 64, 0.1)
    if layers >= 3:
        fill(5248, 4096, math.sqrt(6 / 64))
        fill(9344, 64, 0.1)
    fill(9408, 64, math.sqrt(3 / 64))
    fill(9472, 1, 0.1)
    return p


# input normalisation of the networks: densities of several overlapping boards,
# positions in the unit cube, the sun near the zenith
MEAN = np.array([4.0] * 12 + [0.5] * 3 + [0.9], np.float32)
STDDEV = np.array([5.0] * 12 + [0.2] * 3 + [0.1], np.float32)


def _rows(rng, n):
    """Feature rows as samples of a cloud give them (densities falling off
    along the sun direction) and the optical depths that go with them."""
    base = 8.0 * rng.random((n, 1)) ** 2
    fall = np.exp(-rng.uniform(0.0, 0.4, (n, 1)) * np.arange(12)[None, :])
    f = np.empty((n, NIN), np.float32)
    f[:, :12] = base * fall * rng.uniform(0.7, 1.3, (n, 12))
    f[:, 12:15] = rng.uniform(0.1, 0.9, (n, 3))
    f[:, 15] = rng.uniform(0.8, 1.0, n)
    tau = (0.02 * f[:, :12].sum(axis=1) * rng.uniform(0.9, 1.1, n)).astype(np.float32)
    return f, tau


def _batch_scene(case, seed):
    shape = np.random.default_rng(case["scene"])  # sizes are the case's, boards the seed's
    rng = _rng(case, seed)
    dims = [d for d in (64, 96, 128, 192, 256) if d <= case["max_dim"]]
    clouds = []
    for _ in range(case["clouds"]):
        dim = int(shape.choice(dims))
        n = int(shape.integers(256, case["max_boards"] + 1))
        clouds.append(dict(dim=dim, mips=int(math.log2(dim)) + 1, fmt="rgba32f",
                           boards=_boards(rng, n, 0.5)))
    views = []
    for v in range(case["views"]):
        w, h = ((256, 256), (512, 512), (960, 540), (1920, 1080))[int(shape.integers(4))]
        s = min(1.0, math.sqrt(case["max_pixels"] / (w * h)))
        views.append(dict(cloud=v % case["clouds"],
                          cam=_camera(rng, max(16, int(w * s)), max(16, int(h * s)))))
    return clouds, views


def _compat_scene(case, seed):
    rng = _rng(case, seed)
    n = case["boards"]
    pos = rng.uniform(-2.5, 2.5, (n, 3)).astype(np.float32)
    rad = rng.uniform(1.0, 2.5, n).astype(np.float32)
    a, h = rng.uniform(0, 2 * math.pi), rng.uniform(1.0, 6.0)
    eye = (COMPAT_POS[0] + 14 * math.sin(a), COMPAT_POS[1] + h, COMPAT_POS[2] - 14 * math.cos(a))
    cam = dict(eye=tuple(map(float, eye)), target=COMPAT_POS, fov=60.0, width=case["width"],
               height=case["height"])
    return pos, rad, cam


class _Image(cloudgb.DeviceBuffer):
    """A torch tensor as the library's device destination."""

    def __init__(self, tensor):
        self.tensor = tensor
        self.nbytes = tensor.numel() * tensor.element_size()
        self.ptr = ctypes.c_void_p(tensor.data_ptr())

    def free(self):
        self.ptr = None


def _image(w, h):
    return _Image(torch.zeros((h, w, 4), dtype=torch.float32, device="cuda"))


def _volume(scene, boards=None):
    fmt = cloudgb.FORMAT_RGBA32F if scene["fmt"] == "rgba32f" else cloudgb.FORMAT_BF16_FP16
    vol = cloudgb.CloudVolume(scene["dim"], (-0.5, 0.5), CENTRE, scene["mips"], fmt=fmt)
    if boards is not None:
        vol.set_billboards(*boards)
    return vol


def _shader(case, **more):
    return cloudgb.ConeTraceShader(
        viewSteps=case.get("view_steps", 64), vctSteps=case["sun_steps"],
        vctConeAngle=2.0 * case["half"], vctConeInitialHeight=CONE_H0,
        vctConeMinRadius=MIN_RADIUS, densityScale=case["sigma"], ambient=AMBIENT,
        numOctaves=case.get("octaves", 0), noiseSeed=NOISE["seed"], noiseFrequency=NOISE["freq"],
        freqStep=NOISE["lac"], persStep=NOISE["gain"], **more)


def _gpu_camera(c):
    return cloudgb.Camera(c["eye"], c["target"], fov_y_degrees=c["fov"], width=c["width"],
                          height=c["height"])


def _network(layers, rng, vol=None, shader=None):
    net = surrogate.SunMLP(cloudgb.default_context(), hidden_layers=layers)
    if vol is not None:
        net.configure_for(vol, shader)
    net.configure(mean=MEAN, stddev=STDDEV, tau_scale=TAU_SCALE, feature_min=[-1e6] * NIN,
                  feature_max=[1e6] * NIN)
    net.set_params(_net_params(layers, rng))
    return net


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    rng = _rng(case, seed)
    if kind in ("infer", "gradient", "train"):
        s["net"] = _network(case["layers"], _rng(case, seed, 1))
        f, tau = _rows(rng, case["n"])
        s["f"] = torch.from_numpy(f).cuda()
        s["tau"] = torch.from_numpy(tau).cuda()
        s["out"] = torch.zeros(case["n"], dtype=torch.float32, device="cuda")
        return s
    if kind == "compat":
        pos, rad, cam = _compat_scene(case, seed)
        vol = cloudgb.CloudVolume(case["dim"], (-5.0, 5.0), COMPAT_POS, case["mips"])
        vol.set_billboards(pos, rad)
        vol.update()
        cloudgb.VoxelizeShader().voxelize(vol, cloudgb.Sun(COMPAT_SUN, *COMPAT_MAP))
        s.update(vol=vol, shader=cloudgb.CompatShader(), cam=_gpu_camera(cam),
                 out=_image(cam["width"], cam["height"]))
        return s
    sun = cloudgb.Sun(SUN, *SUN_MAP)
    s["sun"] = sun
    if kind == "batch":
        clouds, views = _batch_scene(case, seed)
        vols = [_volume(c, c["boards"]) for c in clouds]
        for v in vols:
            v.update()
        outs = [_image(v["cam"]["width"], v["cam"]["height"]) for v in views]
        shader = _shader(dict(sun_steps=24, half=0.03, sigma=2.0, view_steps=64, octaves=0))
        s["vols"], s["outs"] = vols, outs
        s["graph"] = cloudgb.FrameGraph(
            cloudgb.default_context(), vols, sun,
            [(vols[v["cloud"]], _gpu_camera(v["cam"]), o) for v, o in zip(views, outs)], shader)
        return s
    vol = _volume(case, _boards(rng, case["boards"], case["rscale"]))
    s["vol"] = vol
    s["shader"] = _shader(case)
    if kind in ("frame", "render", "samples"):
        s["cam"] = _gpu_camera(_camera(rng, case["width"], case["height"]))
    if kind in ("frame", "render"):
        s["out"] = _image(case["width"], case["height"])
        if case["layers"]:
            s["net"] = _network(case["layers"], _rng(case, seed, 1), vol, s["shader"])
            s["shader"] = _shader(case, useMlp=True, mlp=s["net"])
    if kind in ("voxelize", "cones"):
        s["pos"] = torch.from_numpy(_probes(rng, case["n"], case["dim"])).cuda()
        s["out"] = torch.zeros(case["n"], dtype=torch.float32, device="cuda")
        s["params"] = s["shader"].params()
    if kind == "samples":
        s["net"] = _network(3, _rng(case, seed, 1), vol, s["shader"])
        s["host"] = [np.zeros((case["n"], 3), np.float32), np.zeros(case["n"], np.float32)]
    if kind in ("render", "cones", "samples"):
        vol.update()
        cloudgb.VoxelizeShader().voxelize(vol, sun)
    return s


# ---- one pass ----------------------------------------------------------------


def _cones(s):
    """Exact sun cones at the state's device positions, into its device output."""
    d = (ctypes.c_float * 3)(*s["sun"].direction)
    _lib.check(_lib.load().cg_trace_cones(s["vol"].handle, _ptr(s["pos"]), s["case"]["n"], d,
                                          ctypes.byref(s["params"]), _ptr(s["out"]), 1, None),
               "cg_trace_cones")
    return s["out"]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "frame":
        s["vol"].update()
        cloudgb.VoxelizeShader().voxelize(s["vol"], s["sun"])
        return s["shader"].coneTrace(s["vol"], s["cam"], out=s["out"]).tensor
    if kind in ("render", "compat"):
        return s["shader"].coneTrace(s["vol"], s["cam"], out=s["out"]).tensor
    if kind == "voxelize":
        s["vol"].update()
        cloudgb.VoxelizeShader().voxelize(s["vol"], s["sun"])
        return _cones(s)
    if kind == "cones":
        return _cones(s)
    if kind == "batch":
        for v in s["vols"]:
            v.update()
        s["graph"].launch()
        return [o.tensor for o in s["outs"]]
    if kind == "samples":
        p, w = s["host"]
        params, cam, count = s["shader"].params(), s["cam"]._c(), ctypes.c_int()
        _lib.check(_lib.load().cg_march_samples(
            s["vol"].ctx.handle, s["vol"].handle, ctypes.byref(cam), ctypes.byref(params),
            p.ctypes.data_as(_lib.FP), w.ctypes.data_as(_lib.FP), case["n"],
            ctypes.byref(count)), "cg_march_samples")
        tau = s["shader"].traceCone(s["vol"], p, s["sun"].direction)
        return [p, w, tau, s["net"].features(s["vol"], p, s["sun"].direction)]
    net, lib = s["net"], _lib.load()
    if kind == "infer":
        _lib.check(lib.cg_mlp_infer(net.handle, _ptr(s["f"]), case["n"], _ptr(s["out"]), 1, None),
                   "cg_mlp_infer")
        return s["out"]
    if kind == "gradient":
        g, loss = np.empty(NPARAM, np.float32), ctypes.c_float()
        _lib.check(lib.cg_mlp_gradient(net.handle, _ptr(s["f"]), _ptr(s["tau"]), case["n"], SIGMA,
                                       g.ctypes.data_as(_lib.FP), ctypes.byref(loss), 1),
                   "cg_mlp_gradient")
        return [g, float(loss.value)]
    tp = _lib.cg_train_params()
    lib.cg_train_params_default(ctypes.byref(tp))
    tp.steps, tp.batch, tp.sigma, tp.seed = case["steps"], case["batch"], SIGMA, 1
    losses = np.empty(case["steps"], np.float32)
    _lib.check(lib.cg_mlp_train(net.handle, _ptr(s["f"]), _ptr(s["tau"]), case["n"],
                                ctypes.byref(tp), losses.ctypes.data_as(_lib.FP)), "cg_mlp_train")
    params, m, v, _ = net.get_params()
    return [losses, params, m, v]


# ---- what a pass cannot do without -------------------------------------------

TRI = 35   # operations of one trilinear sample: coordinates, weights, seven blends


def _view_work(view, scene, layers):
    """Samples in the cloud from its silhouette (a ball around the centre) and
    the mean chord through it, one cone or one inference each."""
    rb = BALL + 0.5 * sum(RADII) * scene["rscale"]
    half = rb / EYE_DISTANCE / math.tan(math.radians(30.0))
    px = view["width"] * view["height"]
    hit = min(1.0, 0.25 * math.pi * half * half * view["height"] / view["width"])
    n = px * hit * view["view_steps"] * (4 / 3 * rb / 1.2)
    per = TRI + 45 * view["octaves"] + 20
    if layers:
        per += 12 * TRI + 2 * (16 * 64 + (layers - 1) * 64 * 64 + 64) + 5 * 64 * layers
    else:
        per += (TRI + 8) * view["sun_steps"] * 0.7
    return 16.0 * px, n * per


def _volume_bytes(scene):
    fill = 4 / 3 * math.pi * (BALL + 0.5 * sum(RADII) * scene["rscale"]) ** 3
    return scene["dim"] ** 3 * 8 / 7 * min(1.0, fill) * (8 if scene["fmt"] == "rgba32f" else 4)


def _splat_work(scene, boards):
    r = 0.5 * sum(RADII) * scene["rscale"] * scene["dim"]
    texels = boards * math.pi * (0.5 * sum(RADII) * scene["rscale"] / 2.0) ** 2 * SUN_MAP[0] * SUN_MAP[1]
    return (2 * _volume_bytes(scene) + 45.0 * boards + 24.0 * SUN_MAP[0] * SUN_MAP[1],
            boards * 4 / 3 * math.pi * r ** 3 * 4 + texels * 15)


def work(case):
    kind = case["kind"]
    if kind in ("infer", "gradient", "train"):
        net = 2.0 * (16 * 64 + (case["layers"] - 1) * 64 * 64 + 64) + 5 * 64 * case["layers"]
        if kind == "infer":
            return {"bytes": 68.0 * case["n"], "flops": case["n"] * net}
        rows = case["n"] if kind == "gradient" else case["batch"] * case["steps"]
        steps = 1 if kind == "gradient" else case["steps"]
        return {"bytes": 68.0 * rows + 28.0 * NPARAM * steps, "flops": 3 * net * rows}
    if kind == "compat":
        # boards of radius 1.75 at distance 14, a noise march of about eight steps of
        # four octaves and a 16-step cone at each covered pixel until it is opaque
        px = case["width"] * case["height"]
        cover = math.pi * (1.75 / 14 / math.tan(math.radians(30.0)) * case["height"] / 2) ** 2
        return {"bytes": 16.0 * px + case["dim"] ** 3 * 4 + 32 ** 3 * 2,
                "flops": cover * min(case["boards"], 40) * (8 * 4 * 2 * TRI + 16 * 2 * TRI)}
    if kind == "batch":
        b = f = 0.0
        clouds, views = _batch_scene(case, 0)
        for c in clouds:
            x, y = _splat_work(dict(c, rscale=0.5), len(c["boards"][1]))
            b, f = b + x, f + y
        for v in views:
            x, y = _view_work(dict(v["cam"], view_steps=64, octaves=0, sun_steps=24),
                              dict(clouds[v["cloud"]], rscale=0.5), 0)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    if kind in ("cones", "voxelize"):
        b, f = 16.0 * case["n"], case["n"] * case["sun_steps"] * 0.6 * (TRI + 8)
        if kind == "voxelize":
            x, y = _splat_work(case, case["boards"])
            return {"bytes": b + x, "flops": f + y}
        return {"bytes": b + _volume_bytes(case) / 64, "flops": f}
    b, f = _view_work(case, case, case.get("layers", 0))
    b += _volume_bytes(case)
    if kind == "frame":
        x, y = _splat_work(case, case["boards"])
        b, f = b + x, f + y
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits -----------------------------------------------------
# Plain torch.  What decides an index (the sun-view depths and the highlight
# voxels) is defined in 32-bit steps and stays so; coverage is whole numbers.

F32 = np.float32


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _normalize32(v):
    inv = F32(1.0) / np.sqrt(F32(F32(v[0] * v[0] + v[1] * v[1]) + v[2] * v[2]), dtype=F32)
    return [F32(x * inv) for x in v]


def _cross32(a, b):
    return [F32(F32(a[1] * b[2]) - F32(b[1] * a[2])), F32(F32(a[2] * b[0]) - F32(b[2] * a[0])),
            F32(F32(a[0] * b[1]) - F32(b[0] * a[1]))]


def _dot32(a, b):
    return F32(F32(F32(a[0] * b[0]) + F32(a[1] * b[1])) + F32(a[2] * b[2]))


class _Exact:
    """Density R and highlight G levels of a voxelized volume, in 64 bits."""

    def __init__(self, dim, bound, position, mips, boards, sun, sun_map):
        self.dev, self.D, self.L = _device(), dim, mips
        self.pos = [F32(x) for x in position]
        self.wmin = [F32(p - F32(bound)) for p in self.pos]
        self.range = [F32(F32(p + F32(bound)) - w) for p, w in zip(self.pos, self.wmin)]
        self.bound = F32(bound)
        offsets, radii, dens = boards
        self.c = np.stack([self.pos[a] + offsets[:, a] for a in range(3)], axis=1).astype(F32)
        self.r = radii
        R = self._coverage(dens).to(torch.float64) / 65536.0
        G = self._highlights(sun, sun_map)
        self.levels = [(R, G)]
        for _ in range(1, mips):
            R, G = self._halve(R), self._halve(G)
            self.levels.append((R, G))
        self.pad = {}

    @staticmethod
    def _halve(x):
        n = max(1, x.shape[0] // 2)
        return x[:2 * n, :2 * n, :2 * n].reshape(n, 2, n, 2, n, 2).mean(dim=(1, 3, 5))

    def _coverage(self, dens):
        D, Q = self.D, 1 << 20
        v = (self.c.astype(np.float64) - np.array(self.wmin, np.float64)) / np.array(
            self.range, np.float64) * D
        q = np.rint(v * Q).astype(np.int64)
        rq = np.rint(self.r.astype(np.float64) / float(self.range[0]) * D * Q).astype(np.int64)
        r2 = rq * rq
        thr = r2 - (r2 + 9999) // 10000
        dq = np.rint(dens.astype(np.float64) * 65536.0).astype(np.int64)
        lo = np.clip(-((-(q - rq[:, None] - Q // 2)) // Q), 0, D)
        hi = np.clip((q + rq[:, None] - Q // 2) // Q, -1, D - 1) + 1
        out = torch.zeros((D, D, D), dtype=torch.int64, device=self.dev)
        centre = (2 * torch.arange(D, dtype=torch.int64, device=self.dev) + 1) * (Q // 2)
        for b in range(len(thr)):
            if (lo[b] >= hi[b]).any():
                continue
            x, y, z = ((centre[lo[b][a]:hi[b][a]] - int(q[b][a])) ** 2 for a in range(3))
            d2 = z[:, None, None] + y[None, :, None] + x[None, None, :]
            out[lo[b][2]:hi[b][2], lo[b][1]:hi[b][1], lo[b][0]:hi[b][0]] += \
                (d2 <= int(thr[b])) * int(dq[b])
        return out

    def _highlights(self, sun, sun_map):
        W, H = sun_map
        d = np.asarray(sun, np.float64)
        d = d / np.sqrt((d * d).sum())
        look = _normalize32([F32(-F32(x)) for x in d])
        dist = np.sqrt(F32(F32(self.bound * self.bound * 1 + self.bound * self.bound) +
                           self.bound * self.bound), dtype=F32)
        eye = [F32(p - F32(x * dist)) for p, x in zip(self.pos, look)]
        f = _normalize32([F32(p - e) for p, e in zip(self.pos, eye)])
        right = _normalize32(_cross32(f, [F32(0), F32(1), F32(0)]))
        up = _cross32(right, f)
        t = [F32(-_dot32(right, eye)), F32(-_dot32(up, eye)), _dot32(f, eye)]
        span_lo, span_hi = F32(-2) * self.bound, F32(2) * self.bound
        near = F32(0.01)
        dev = self.dev

        def whole(x):  # on the device: a division by a host number would be rounded twice
            return torch.full((), float(x), dtype=torch.float32, device=dev)

        def texels(n):
            i = torch.arange(n, dtype=torch.float32, device=dev) + 0.5
            return float(span_lo) + (i / whole(n)) * float(F32(span_hi - span_lo))

        X, Y = texels(W), texels(H)
        c = self.c

        def row(m, shift):
            return ((m[0] * c[:, 0] + m[1] * c[:, 1]) + m[2] * c[:, 2]) + shift

        nf = [F32(-x) for x in f]
        view = np.stack([row(right, t[0]), row(up, t[1]), row(nf, t[2])], axis=1)
        radii = torch.from_numpy(self.r).to(dev)
        empty = torch.iinfo(torch.int64).max
        keys = torch.full((H, W), empty, dtype=torch.int64, device=dev)
        zmap = torch.zeros((H, W), dtype=torch.float32, device=dev)
        scale = 1.0 / (float(span_hi) - float(span_lo))
        for k in range(len(c)):
            r = float(self.r[k])
            if r <= 0:
                continue
            i0 = max(0, int(((view[k][0] - r) - span_lo) * scale * W) - 3)
            i1 = min(W, int(((view[k][0] + r) - span_lo) * scale * W) + 4)
            j0 = max(0, int(((view[k][1] - r) - span_lo) * scale * H) - 3)
            j1 = min(H, int(((view[k][1] + r) - span_lo) * scale * H) + 4)
            if i0 >= i1 or j0 >= j1:
                continue
            x, y = X[i0:i1][None, :], Y[j0:j1][:, None]
            dx, dy = x - float(view[k][0]), y - float(view[k][1])
            q = torch.sqrt(dx * dx + dy * dy) / radii[k]
            prof = torch.sqrt(torch.clamp(1.0 - q * q, min=0.0))
            zs = float(view[k][2]) + r * prof
            dz = zs + float(near)
            depth = torch.sqrt((x * x + y * y) + dz * dz)
            key = (depth.view(torch.int32).to(torch.int64) << 32) | k
            old = keys[j0:j1, i0:i1]
            win = (prof >= float(F32(0.01))) & (key < old)
            keys[j0:j1, i0:i1] = torch.where(win, key, old)
            zmap[j0:j1, i0:i1] = torch.where(win, zs, zmap[j0:j1, i0:i1])
        G = torch.zeros(self.D ** 3, dtype=torch.float64, device=dev)
        jj, ii = torch.nonzero(keys != empty, as_tuple=True)
        x, y, z = X[ii], Y[jj], zmap[jj, ii]
        p = [((x * float(right[a]) + y * float(up[a])) + z * float(-f[a])) + float(eye[a])
             for a in range(3)]
        step = min(F32(r / F32(self.D)) for r in self.range)
        o = float(F32(step * F32(0.57735026)))
        for k in range(-1, 8):
            ids, ok = [], torch.ones_like(x, dtype=torch.bool)
            for a, bit in enumerate((4, 2, 1)):
                pa = p[a] if k < 0 else (p[a] - o if k & bit else p[a] + o)
                v = ((pa - float(self.wmin[a])) / whole(self.range[a])) * float(self.D)
                ok &= (v > -1.0) & (v < float(self.D))
                ids.append(v.to(torch.int64))
            at = ((ids[2] * self.D + ids[1]) * self.D + ids[0])[ok]
            G[at] = 1.0
        return G.reshape(self.D, self.D, self.D)

    def tri(self, l, p, channel, border):
        """Trilinear samples of level l at level-0 positions p (three vectors)."""
        key = (l, channel, border)
        if key not in self.pad:
            x = self.levels[l][channel]
            if border:
                x = torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1))
            self.pad[key] = x.contiguous()
        x = self.pad[key]
        N, n = self.levels[l][0].shape[0], x.shape[0]
        sc = N / self.D
        lo, hi, w = [], [], []
        for a in range(3):
            u = p[a] * sc - 0.5
            f = torch.floor(u)
            w.append(u - f)
            i = f.to(torch.int64) + (1 if border else 0)
            lo.append(i.clamp(0, n - 1))
            hi.append((i + 1).clamp(0, n - 1))
        flat = x.reshape(-1)
        zz = (lo[2] * n * n, hi[2] * n * n)
        yy = (lo[1] * n, hi[1] * n)
        out = 0.0
        for c, wz in ((0, 1 - w[2]), (1, w[2])):
            for b, wy in ((0, 1 - w[1]), (1, w[1])):
                at = zz[c] + yy[b]
                out = out + wz * wy * ((1 - w[0]) * flat[at + lo[0]] + w[0] * flat[at + hi[0]])
        return out

    def quad(self, p, l0, frac, channel, border):
        v = self.tri(l0, p, channel, border)
        if l0 + 1 < self.L:
            v = v + frac * (self.tri(l0 + 1, p, channel, border) - v)
        return v

    def cone(self, p, s, steps, half, h0, rmin):
        """Optical depth of the transmittance cone (floored radius)."""
        tan, vw, h, tau = math.tan(float(F32(half))), float(self.range[0]) / self.D, h0, 0.0
        for _ in range(steps):
            r = max(h * tan, rmin)
            lod = min(math.log2(max(1.0, 2 * r)), self.L - 1.0)
            l0 = int(lod)
            tau = tau + r * vw * self.quad([p[a] + h * s[a] for a in range(3)], l0, lod - l0, 0,
                                           True)
            h += r
        return tau

    def reference_cone(self, p, s, steps, angle, h0):
        """The reference's weighted sum of the light channel."""
        tan, h, acc = math.tan(float(F32(angle)) / 2), h0, 0.0
        for i in range(steps):
            r = h * tan
            lod = min(max(math.log2(max(1.0, 2 * r)), 0.0), self.L - 1.0)
            l0 = int(lod)
            acc = acc + (i + 1) / steps * self.quad([p[a] + h * s[a] for a in range(3)], l0,
                                                    lod - l0, 1, False)
            h += r
        return acc


def _unit(v):
    v = np.asarray(v, np.float64)
    return v / np.sqrt((v * v).sum())


def _lattice(octave, lo, n, dev):
    """PCG3D lattice values (n^3 from lo) of one octave."""
    M = 0xFFFFFFFF
    k = (NOISE["seed"] * 0x9E3779B9 + octave * 0x85EBCA6B + 1) & M
    g = torch.arange(lo, lo + n, dtype=torch.int64, device=dev)
    x = ((g + k) & M)[None, None, :].expand(n, n, n)
    y = ((g + (k ^ 0x68E31DA4)) & M)[None, :, None].expand(n, n, n)
    z = ((g + (k ^ 0xB5297A4D)) & M)[:, None, None].expand(n, n, n)
    x, y, z = ((u * 1664525 + 1013904223) & M for u in (x, y, z))
    x = (x + y * z) & M
    y = (y + z * x) & M
    z = (z + x * y) & M
    x, y, z = (u ^ (u >> 16) for u in (x, y, z))
    return (((x + y * z) & M) >> 8).to(torch.float64) / 16777216.0


class _Noise:
    def __init__(self, octaves, dev):
        self.tabs = []
        for o in range(octaves):
            n = int(NOISE["freq"] * NOISE["lac"] ** o) + 5
            self.tabs.append(_lattice(o, -2, n, dev))

    def __call__(self, p):
        if not self.tabs:
            return 1.0
        amp, total, norm, f = 1.0, 0.0, 0.0, NOISE["freq"]
        for t in self.tabs:
            n, idx, w = t.shape[0], [], []
            for a in range(3):
                u = p[a] * f
                i = torch.floor(u)
                d = u - i
                w.append(d * d * (3 - 2 * d))
                idx.append((i.to(torch.int64) + 2).clamp(0, n - 2))
            flat, v = t.reshape(-1), 0.0
            for c in (0, 1):
                for b in (0, 1):
                    at = ((idx[2] + c) * n + idx[1] + b) * n + idx[0]
                    wz = w[2] if c else 1 - w[2]
                    wy = w[1] if b else 1 - w[1]
                    v = v + wz * wy * ((1 - w[0]) * flat[at] + w[0] * flat[at + 1])
            total, norm = total + amp * v, norm + amp
            amp, f = amp * NOISE["gain"], f * NOISE["lac"]
        return total / norm


def _net_exact(layers, params, f):
    """The network's optical depth for feature rows f, in 64 bits."""
    p = params if torch.is_tensor(params) else torch.from_numpy(params).to(f.device, torch.float64)
    dev = f.device
    x = (f - torch.from_numpy(MEAN).to(dev, torch.float64)) / torch.from_numpy(STDDEV).to(
        dev, torch.float64)
    for w, b, k in ((0, 1024, 16), (1088, 5184, 64), (5248, 9344, 64))[:layers]:
        x = torch.nn.functional.silu(x @ p[w:w + 64 * k].reshape(64, k).T + p[b:b + 64])
    return TAU_SCALE * torch.nn.functional.softplus(x @ p[9408:9472] + p[9472])


def _rays(cam, dev):
    f = _unit(np.asarray(cam["target"], np.float32).astype(np.float64) -
              np.asarray(cam["eye"], np.float32).astype(np.float64))
    s = _unit(np.cross(f, (0.0, 1.0, 0.0)))
    u = np.cross(s, f)
    W, H, t = cam["width"], cam["height"], math.tan(math.radians(cam["fov"]) / 2)
    x = (2 * (torch.arange(W, dtype=torch.float64, device=dev) + 0.5) / W - 1) * t * W / H
    y = (1 - 2 * (torch.arange(H, dtype=torch.float64, device=dev) + 0.5) / H) * t
    x, y = x[None, :].expand(H, W).reshape(-1), y[:, None].expand(H, W).reshape(-1)
    return f, s, u, x, y, t


def _render_exact(ex, cam, view, sigma, net=None):
    dev = ex.dev
    f, s, u, X, Y, tan = _rays(cam, dev)
    eye = np.asarray(cam["eye"], np.float32).astype(np.float64)
    W, H, Nv = cam["width"], cam["height"], view["view_steps"]
    noise, sun = _Noise(view["octaves"], dev), _unit(SUN)
    out = torch.zeros((H * W, 4), dtype=torch.float64, device=dev)
    lo = [float(x) for x in ex.wmin]
    rng = [float(x) for x in ex.range]
    pixk = tan / H * ex.D / rng[0]
    for at in range(0, H * W, 1 << 19):
        x, y = X[at:at + (1 << 19)], Y[at:at + (1 << 19)]
        d = [f[a] + x * s[a] + y * u[a] for a in range(3)]
        inv = 1 / torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
        d = [v * inv for v in d]
        tin, tout = torch.zeros_like(x), torch.full_like(x, 1e30)
        for a in range(3):
            t0, t1 = (lo[a] - eye[a]) / d[a], (lo[a] + rng[a] - eye[a]) / d[a]
            tin = torch.maximum(tin, torch.minimum(t0, t1))
            tout = torch.minimum(tout, torch.maximum(t0, t1))
        hit = torch.nonzero(tout > tin).reshape(-1)
        if not hit.numel():
            continue
        d, tin = [v[hit] for v in d], tin[hit]
        dt = (tout[hit] - tin) / Nv
        T, C = torch.ones_like(tin), torch.zeros_like(tin)
        for k in range(Nv):
            t = tin + (k + 0.5) * dt
            p = [eye[a] + t * d[a] for a in range(3)]
            v = [(p[a] - lo[a]) * (ex.D / rng[a]) for a in range(3)]
            lod = torch.log2(torch.clamp(2 * t * pixk, min=1.0)).clamp(max=ex.L - 1.0)
            R = torch.zeros_like(t)
            l0 = lod.to(torch.int64)
            for l in torch.unique(l0).tolist():
                m = torch.nonzero((l0 == l) & (T >= CUTOFF)).reshape(-1)
                R[m] = ex.quad([q[m] for q in v], l, lod[m] - l, 0, True)
            m = torch.nonzero(R > 0).reshape(-1)
            if not m.numel():
                continue
            vm, pm, lm = [q[m] for q in v], [q[m] for q in p], l0[m]
            rho = R[m] * noise(pm)
            G = torch.zeros_like(rho)
            for l in torch.unique(lm).tolist():
                g = torch.nonzero(lm == l).reshape(-1)
                G[g] = ex.quad([q[g] for q in vm], l, lod[m][g] - l, 1, True)
            alpha = 1 - torch.exp(-sigma * rho * dt[m])
            if net is None:
                tau = ex.cone(vm, sun, view["sun_steps"], view["half"], CONE_H0, MIN_RADIUS)
            else:
                tau = _net_exact(net[0], net[1], _features_exact(ex, vm, sun))
            light = torch.exp(-sigma * tau) * (AMBIENT + (1 - AMBIENT) * G)
            C[m] += T[m] * alpha * light
            T[m] *= 1 - alpha
        out[at + hit] = torch.stack([C, C, C, 1 - T], dim=1)
    return out.reshape(H, W, 4)


def _features_exact(ex, v, sun):
    lb = int(math.floor(math.log2(max(1.0, 2 * MIN_RADIUS))))
    cols = []
    for i in range(4):
        for k in range(3):
            d = CONE_H0 + (k + 0.5) * 2 ** (lb + i)
            cols.append(ex.tri(min(lb + i, ex.L - 1), [v[a] + d * sun[a] for a in range(3)], 0,
                               True))
    cols += [v[a] / ex.D for a in range(3)] + [torch.full_like(v[0], sun[1])]
    return torch.stack(cols, dim=1)


def _noise_map(dev):
    """Green and alpha of the compat noise map (seed 1), decoded, [z, y, x]."""
    n, M = 32, (1 << 64) - 1
    st = (1 * 0x2545F4914F6CDD1D + 0x632BE59BD9B4E019) & M
    a = np.empty(n ** 3, np.int64)
    for i in range(n ** 3):
        st = (st + 0x9E3779B97F4A7C15) & M
        z = ((st ^ (st >> 30)) * 0xBF58476D1CE4E5B9) & M
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M
        a[i] = ((z ^ (z >> 31)) >> 56) - 128
    a = a.reshape(n, n, n)
    g = [np.roll(a, -1, ax) - 2 * np.roll(a, 1, ax) for ax in (2, 1, 0)]
    S = g[0] ** 2 + g[1] ** 2 + g[2] ** 2
    c = np.floor(np.sqrt(16384.0 * g[1] ** 2 / np.maximum(S, 1))).astype(np.int64)
    c = np.where(c * c * S > 16384 * g[1] ** 2, c - 1, c)
    c = np.where((c + 1) ** 2 * S <= 16384 * g[1] ** 2, c + 1, c)
    c = np.where(S == 0, 0, np.minimum(c, 127)) * np.sign(g[1])
    return (torch.from_numpy(c / 127.0).to(dev),
            torch.from_numpy(np.maximum(a / 127.0, -1.0)).to(dev))


def _compat_exact(ex, cam):
    dev = ex.dev
    f, s, u, X, Y, _ = _rays(cam, dev)
    W, H = cam["width"], cam["height"]
    eye = np.asarray(cam["eye"], np.float32).astype(np.float64)
    green, alpha = (t.reshape(-1) for t in _noise_map(dev))
    sun = _unit(COMPAT_SUN)
    out = torch.tensor([0.2, 0.3, 0.5, 1.0], dtype=torch.float64, device=dev).repeat(H * W, 1)

    def tap(q):
        lo, hi, w = [], [], []
        for a in range(3):
            t = q[a] * 32 - 0.5
            i = torch.floor(t)
            w.append(t - i)
            i = i.to(torch.int64) % 32
            lo.append(i)
            hi.append((i + 1) % 32)
        g = al = 0.0
        for c, wz in ((lo, 1 - w[2]), (hi, w[2])):
            for b, wy in ((lo, 1 - w[1]), (hi, w[1])):
                at = (c[2] * 32 + b[1]) * 32
                for e, wx in ((lo, 1 - w[0]), (hi, w[0])):
                    k = wz * wy * wx
                    g, al = g + k * green[at + e[0]], al + k * alpha[at + e[0]]
        return g, al

    c64, r64 = ex.c.astype(np.float64), ex.r.astype(np.float64)
    dist = ((c64 - eye) ** 2).sum(axis=1)
    tan = math.tan(math.radians(cam["fov"]) / 2)
    for b in sorted(range(len(dist)), key=lambda i: (-dist[i], -i)):
        c, r = c64[b], r64[b]
        o = c - eye
        z = float(o @ f)
        if not 0.01 < z < 2500 or r <= 0:
            continue
        # the quad's pixels, from its rectangle on the view plane
        cols = [((float(o @ s) + e * r) / z / (tan * W / H) + 1) * W / 2 - 0.5 for e in (-1, 1)]
        rows = [(1 - (float(o @ u) + e * r) / z / tan) * H / 2 - 0.5 for e in (1, -1)]
        i0, i1 = max(0, int(cols[0]) - 1), min(W, int(cols[1]) + 3)
        j0, j1 = max(0, int(rows[0]) - 1), min(H, int(rows[1]) + 3)
        if i0 >= i1 or j0 >= j1:
            continue
        at = (torch.arange(j0, j1, device=dev)[:, None] * W +
              torch.arange(i0, i1, device=dev)[None, :]).reshape(-1)
        px = [eye[a] + z * (f[a] + X[at] * s[a] + Y[at] * u[a]) for a in range(3)]
        x = sum((px[a] - c[a]) * s[a] for a in range(3)) / r
        y = sum((px[a] - c[a]) * u[a] for a in range(3)) / r
        d2 = r * r * (x * x + y * y)
        sc2 = 1 - d2 / (r * r)
        disc = 4 * (r * r - d2)
        on = torch.nonzero((x.abs() <= 1) & (y.abs() <= 1) & (disc >= 0.01) &
                           (torch.sqrt(sc2.clamp(min=0)) >= 0.01)).reshape(-1)
        if not on.numel():
            continue
        at, px, x, y, disc, sc2 = at[on], [q[on] for q in px], x[on], y[on], disc[on], sc2[on]
        half = torch.sqrt(disc) / 2          # the chord's ends lie at -+half along -f
        near = [px[a] + f[a] * half for a in range(3)]
        far = [px[a] - f[a] * half for a in range(3)]
        un = [(near[a] - c[a]) / r for a in range(3)]
        cn = [q / 40.0 for q in near]
        e = [far[a] / 40.0 - cn[a] for a in range(3)]
        steps = torch.clamp(torch.sqrt(e[0] ** 2 + e[1] ** 2 + e[2] ** 2) / float(F32(0.01)),
                            max=6.0) + 2.0
        dl = [q / (steps - 1) for q in e]
        ro = torch.zeros_like(x)
        rl = torch.zeros_like(x)
        for i in range(8):
            m = torch.nonzero(steps > i).reshape(-1)
            if not m.numel():
                break
            cc = [(cn[a] + i * dl[a])[m] for a in range(3)]
            uu = [(un[a] + i * dl[a])[m] for a in range(3)]
            ng = na = 0.0
            for k in range(4):
                g, al = tap([q * 3.0 ** k for q in cc])
                ng, na = ng + 0.5 ** k * g, na + 0.5 ** k * al
            n2 = uu[0] ** 2 + uu[1] ** 2 + uu[2] ** 2
            ng = ng + uu[1] / torch.sqrt(n2)
            ro[m] += na.abs() * (1 - n2)
            rl[m] += torch.clamp(ng * 0.5 + 0.5, 0, 1)
        col = float(F32(0.2)) + float(F32(0.45)) * rl / (steps - 1)
        a = torch.clamp(ro * 4.0 / (steps - 1), 0, 1) * (1 - torch.sqrt((x / 2) ** 2 + (y / 2) ** 2) * 2)
        sc = torch.sqrt(sc2)
        v = [ex.D * ((px[k] - f[k] * r * sc - float(ex.wmin[k])) / float(ex.range[k]))
             for k in range(3)]
        col = torch.clamp(col * ex.reference_cone(v, sun, 16, 0.9, float(F32(0.1))), 0, 1)
        a = torch.clamp(a, 0, 1)
        src = torch.stack([col, col, col, a], dim=1)
        out[at] = src * a[:, None] + out[at] * (1 - a)[:, None]
    return out.reshape(H, W, 4)


def _loss_exact(layers, p, f, tau):
    that = torch.exp(-SIGMA * _net_exact(layers, p, f))
    return ((that - torch.exp(-SIGMA * tau)) ** 2).mean()


def _train_exact(case, seed):
    dev = _device()
    f, tau = (torch.from_numpy(x).to(dev, torch.float64) for x in _rows(_rng(case, seed), case["n"]))
    p = torch.from_numpy(_net_params(case["layers"], _rng(case, seed, 1))).to(dev, torch.float64)
    used = torch.ones(NPARAM, dtype=torch.bool, device=dev)
    if case["layers"] < 3:
        used[{1: 1088, 2: 5248}[case["layers"]]:9408] = False
    if case["kind"] == "gradient":
        p.requires_grad_(True)
        loss = _loss_exact(case["layers"], p, f, tau)
        loss.backward()
        return [p.grad, loss.detach()]
    n, mul = case["n"], 2246822519
    while math.gcd(mul, n) != 1:
        mul += 2
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    losses = []
    for step in range(case["steps"]):
        lin = (step * case["batch"] + torch.arange(case["batch"], device=dev)) % n
        at = (lin * (mul % n)) % n
        p.requires_grad_(True)
        loss = _loss_exact(case["layers"], p, f[at], tau[at])
        g, = torch.autograd.grad(loss, p)
        losses.append(loss.detach())
        with torch.no_grad():
            g = torch.where(used, g, torch.zeros_like(g))
            b1, b2 = float(F32(0.9)), float(F32(0.999))
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            p = p - float(F32(1e-3)) * (m / (1 - b1 ** (step + 1))) / (
                torch.sqrt(v / (1 - b2 ** (step + 1))) + 1e-8)
    return [torch.stack(losses), p.detach(), m, v]


def exact(case, seed):
    kind = case["kind"]
    rng = _rng(case, seed)
    dev = _device()
    if kind == "samples":
        return None  # the order and number of the samples are the renderer's own
    if kind == "infer":
        f, _ = _rows(rng, case["n"])
        net = _net_params(case["layers"], _rng(case, seed, 1))
        return _net_exact(case["layers"], net, torch.from_numpy(f).to(dev, torch.float64))
    if kind in ("gradient", "train"):
        return _train_exact(case, seed)
    if kind == "compat":
        pos, rad, cam = _compat_scene(case, seed)
        ex = _Exact(case["dim"], 5.0, COMPAT_POS, case["mips"],
                    (pos, rad, np.ones(len(rad), np.float32)), COMPAT_SUN, COMPAT_MAP)
        return _compat_exact(ex, cam)
    if kind == "batch":
        clouds, views = _batch_scene(case, seed)
        vols = [_Exact(c["dim"], 0.5, CENTRE, c["mips"], c["boards"], SUN, SUN_MAP)
                for c in clouds]
        view = dict(view_steps=64, octaves=0, sun_steps=24, half=0.03)
        return [_render_exact(vols[v["cloud"]], v["cam"], view, 2.0) for v in views]
    ex = _Exact(case["dim"], 0.5, CENTRE, case["mips"],
                _boards(rng, case["boards"], case["rscale"]), SUN, SUN_MAP)
    if kind in ("voxelize", "cones"):
        p = torch.from_numpy(_probes(rng, case["n"], case["dim"])).to(dev, torch.float64)
        return ex.cone([p[:, a] for a in range(3)], _unit(SUN), case["sun_steps"], case["half"],
                       CONE_H0, MIN_RADIUS)
    cam = _camera(rng, case["width"], case["height"])
    net = (case["layers"], _net_params(case["layers"], _rng(case, seed, 1))) \
        if case["layers"] else None
    return _render_exact(ex, cam, case, case["sigma"], net)
