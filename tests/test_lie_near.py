"""The near-identity SL(3) retraction against the general one, on the CPU
(fm_lie.cuh compiles for the host).  Both form e^L of the same log L, which
each has to a few roundings: entries are O(1), so 2e-14 leaves room for about
a hundred of them.  The stop test of the log's Newton corrections (residual
below 1e-12) can fall on different sides for a residual next to it; either
side is then within 1e-12 of G, ||G||_F < 3, so such a draw may differ by
3e-12, and there are hardly any."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("lie") / "lie_near_check")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-O2", "-std=c++17", os.path.join(HERE, "cpp", "lie_near_check.cpp"),
                    "-I", os.path.join(HERE, "..", "atlas-flexmesh_b200", "csrc"),
                    "-I", "/usr/local/cuda/include", "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("lim", [1e-12, 9.9e-8, 1.01e-7, 1e-5, 1e-2, 0.124, 0.126, 0.3, 0.4999])
def test_near_matches_general(check, lim):
    worst, inner, flips = subprocess.run([check, str(lim)], check=True, capture_output=True,
                                         text=True).stdout.split()
    assert float(inner) <= 2e-14
    assert float(worst) <= 3e-12 and int(flips) <= 2
