"""The rasteriser's and the lift's division by a known reciprocal and their sign tests
(csrc/tri_test.cuh), compiled for the host, against the correctly rounded quotient: random
operands of every exponent, mantissas of few bits and of many ones, quotients next to
halfway between two doubles.  No GPU needed."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def host_bin(tmp_path_factory):
    gxx, cuda = shutil.which("g++"), "/usr/local/cuda/include"
    if not gxx or not os.path.exists(cuda):
        pytest.skip("no host C++ compiler or no CUDA headers")
    out = str(tmp_path_factory.mktemp("tri") / "tri_test")
    subprocess.run([gxx, "-O2", "-ffp-contract=off", "-std=c++17", "-I", cuda, "-I",
                    os.path.join(ROOT, "surface-remesher_gb300", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "tri_test_host.cpp")], check=True)
    return out


@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_division_by_a_reciprocal_is_correctly_rounded(host_bin, seed):
    r = subprocess.run([host_bin, str(seed), "2000000"], capture_output=True, text=True,
                       check=True).stdout.split()
    assert r[0] == "ok", r
    assert int(r[1]) > 100000
