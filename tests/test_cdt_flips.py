"""The constrained Delaunay stage's flip rounds, replayed on the CPU
(tests/cdt_flips_host.cpp): what a flip that lost its claims reads while the winners
change the mesh stays inside it, and it never takes itself for a winner.  No GPU needed."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def flips_bin(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    out = str(tmp_path_factory.mktemp("cdt_flips") / "flips")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I",
                    os.path.join(ROOT, "surface-remesher_gb300", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "cdt_flips_host.cpp")], check=True)
    return out


@pytest.mark.parametrize("points", [5, 12, 40, 150, 400])
def test_losing_flips_read_inside_the_mesh(flips_bin, points):
    hull = 0
    for seed in range(8):
        r = subprocess.run([flips_bin, str(points), str(seed)], capture_output=True, text=True,
                           check=True).stdout.split()
        assert r[0] == "ok", r
        hull += int(r[2])
    assert hull > 0 or points < 12  # losers whose edge had become a hull edge were among them
