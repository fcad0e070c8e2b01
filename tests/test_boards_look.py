"""The quick look at a board list (csrc/cg_boards.h) on the CPU, built with the
undefined-behaviour sanitizer: no float is out of an integer's range and no sum
overflows, also for radii and positions that are refused."""
import math
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cloud-renderer_gb300", "csrc")
SANITIZE = ["-fsanitize=undefined,float-cast-overflow", "-fno-sanitize-recover=all"]


@pytest.fixture(scope="module")
def boards_exe(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("cpp") / "boards")
    cmd = [os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-Wall", "-Wextra",
           "-ffp-contract=off", *SANITIZE, "-I", CSRC,
           os.path.join(ROOT, "tests", "cpp", "boards.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0 and "ubsan" in r.stderr:
        pytest.skip("no sanitizer runtime")
    assert r.returncode == 0, r.stderr
    return exe


def test_any_board_list_is_defined(boards_exe):
    r = subprocess.run([boards_exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lines = r.stdout.split("\n")[:-1]
    assert len(lines) == 4 * 11 * 5
    for line in lines:
        _, radius, x, fine = line.split()
        radius, x = float(radius), float(x)
        ok = 0 <= radius <= 1 and math.isfinite(x)
        if not ok:
            assert fine == "0", line
        elif radius < 0.5:
            assert fine == "1", line


@pytest.mark.gpu
@pytest.mark.parametrize("radius", [-1e9, -3.4e38, 1e9, 3.4e38])
def test_extreme_radii_are_refused_by_name(ctx, radius):
    import numpy as np

    import cloudgb
    vol = cloudgb.CloudVolume(256, (-0.5, 0.5), (0.5, 0.5, 0.5), 3,
                              fmt=cloudgb.FORMAT_BF16_FP16, ctx=ctx)
    rad = np.full(600, 0.01, np.float32)
    rad[257::2] = radius
    vol.set_billboards(np.zeros((600, 3), np.float32), rad)
    with pytest.raises(Exception, match="billboard 257: "):
        vol.update()
    vol.close()
