"""Board uploads: the records made on the device, what is refused and in which
order, and uploads that follow one another without waiting."""
import numpy as np
import pytest

import cloudgb
from cloudgb import configs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _volume(ctx, dim=40, bounds=(-0.5, 0.5), position=(0.5, 0.5, 0.5)):
    return cloudgb.CloudVolume(dim, bounds, position, 3, ctx=ctx)


def _boards(seed, n, size=1.0, bounds=(-0.5, 0.5)):
    rng = np.random.default_rng(seed)
    lo, hi = bounds
    pos = rng.uniform(lo - 1.5 * size, hi + 1.5 * size, (n, 3)).astype(np.float32)
    inside = rng.random(n) < 0.8
    pos[inside] = rng.uniform(lo, hi, (int(inside.sum()), 3)).astype(np.float32)
    rad = (size * rng.choice([0.0, 1e-4, 0.013, 0.05, 0.21], n)).astype(np.float32)
    return pos, rad, rng.uniform(0.0, 3.0, n).astype(np.float32)


def _coverage(vol):
    cloudgb.VoxelizeShader().voxelize(vol, cloudgb.Sun((0.3, 1.0, 0.2), 24, 16))
    return vol.read_coverage()


@pytest.mark.parametrize("n", [0, 1, 127, 128, 129, 257, 3000])
@pytest.mark.parametrize("bounds,position", [((-0.5, 0.5), (0.5, 0.5, 0.5)),
                                             ((-1.7, 2.0), (-30.0, 0.1, 7.0))])
def test_records_against_the_oracle(ctx, n, bounds, position):
    """Centres in, beside and far outside a volume whose extent is, and is not, a
    power of two; radii from zero; fluffiness: counts and sums bit for bit."""
    size = bounds[1] - bounds[0]
    pos, rad, den = _boards(n, n, size, bounds)
    vol = _volume(ctx, 40, bounds, position)
    vol.fluffiness = 1.3
    vol.set_billboards(pos, rad, den)
    vol.update()
    ov = O.OracleVolume(40, bounds, position, 3)
    assert ov.set_boards(pos, rad, den, 1.3) == 0
    assert ov.voxelize((0.3, 1.0, 0.2), 24, 16) == 0
    cnt, dq = _coverage(vol)
    ocnt, odq = ov.coverage()
    assert np.array_equal(cnt, ocnt)
    assert np.array_equal(dq, odq)


@pytest.mark.parametrize("at", [0, 130, 299])
@pytest.mark.parametrize("what,value,message", [
    ("rad", -1e-9, "radius must be finite"), ("rad", np.nan, "radius must be finite"),
    ("rad", np.inf, "radius must be finite"), ("rad", 1.01, "exceeds the volume extent"),
    ("den", -1.0, "density must be in"), ("den", 32768.0, "density must be in"),
    ("den", np.nan, "density must be in"), ("pos", np.nan, "non-finite position"),
    ("pos", -np.inf, "non-finite position")])
def test_refused_boards(ctx, at, what, value, message):
    """The first refused board is named, and the list in use stays."""
    vol = _volume(ctx)
    vol.set_billboards(*_boards(1, 300))
    vol.update()
    before = _coverage(vol)
    pos, rad, den = _boards(2, 300)
    if at < 299:
        rad[299] = np.nan  # a later fault is not the one named
    dict(pos=pos, rad=rad, den=den)[what][at] = value
    vol.set_billboards(pos, rad, den)
    with pytest.raises(Exception, match=f"billboard {at}: .*{message}"):
        vol.update()
    again = _coverage(vol)
    assert all(np.array_equal(a, b) for a, b in zip(before, again))
    rad[at] = 1.0  # exactly the extent is accepted
    rad[299] = 0.1
    pos[at], den[at] = 0.0, 1.0
    vol.set_billboards(pos, rad, den)
    vol.update()


def test_uploads_in_a_row(ctx):
    """Uploads and voxelizes queued without a wait, lists growing and shrinking,
    on two streams: each volume ends with its last list."""
    torch = pytest.importorskip("torch")
    streams = [None, torch.cuda.Stream().cuda_stream]
    sun = cloudgb.Sun((0.3, 1.0, 0.2), 640, 360)
    vols = [_volume(ctx, 64) for _ in streams]
    for i, n in enumerate([3000, 10, 3000, 2999, 20000, 1, 20000]):
        for vol, stream in zip(vols, streams):
            vol.set_billboards(*_boards(i, n))
            vol.update()
            cloudgb.VoxelizeShader().voxelize(vol, sun, stream=stream)
    torch.cuda.synchronize()
    fresh = _volume(ctx, 64)
    fresh.set_billboards(*_boards(6, 20000))
    fresh.update()
    cloudgb.VoxelizeShader().voxelize(fresh, sun)
    for vol in vols:
        for a, b in zip(vol.read_coverage(), fresh.read_coverage()):
            assert np.array_equal(a, b)
        assert np.array_equal(vol.read_level(0), fresh.read_level(0))
