"""The bounds that size the bars' list of an upload (csrc/cg_boards.h) against the exact
number of board-bar pairs, on the CPU: neither is below it, and that of long lists is
above it only by boards whose ends lie at voxel centres and one for each board that
meets no voxel centre."""
import os
import subprocess

from test_boards_look import CSRC, ROOT, SANITIZE


def test_bound_of_the_pairs(tmp_path):
    exe = str(tmp_path / "bound")
    base = [os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-Wall", "-Wextra",
            "-ffp-contract=off", "-I", CSRC, os.path.join(ROOT, "tests", "cpp", "boards_bound.cpp"),
            "-o", exe]
    r = subprocess.run(base + SANITIZE, capture_output=True, text=True)
    if r.returncode != 0:  # (a compiler without the sanitizer's runtime)
        r = subprocess.run(base, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lines = r.stdout.split("\n")[:-1]
    assert len(lines) == 8 * 2 * 3 * 6
    for line in lines:
        _, size, at, kind, fine, rough, bound, exact, none = line.split()
        kind, bound, exact, none = int(kind), int(bound), int(exact), int(none)
        assert fine == "1", line
        assert int(rough) >= exact and bound >= exact, line
        if kind == 1:  # half of the boards end at voxel centres: a bar more an axis and end
            assert bound <= 8 * exact + none + 1, line
        else:
            # each of the six ends lies within the slack of a centre once in a hundred
            # times; its axis then counts one bar more, so at most twice as many
            assert bound <= 1.1 * exact + none + 40, line
