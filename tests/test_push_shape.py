"""Clusters and warps of the push solves (fm_setup.hpp push_shape) from the level
widths alone: tests/cpp/push_shape_check.cpp prints the choice for level
pointers given as widths.  The expectations are the measured better sides of
the rule, and its caps."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "atlas-flexmesh_b200", "csrc")


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("shape") / "push_shape_check")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", CSRC, "-o", out,
                    os.path.join(ROOT, "tests", "cpp", "push_shape_check.cpp"),
                    os.path.join(CSRC, "fm_setup.cpp")], check=True, timeout=300)

    def run(fwd, bwd=None, available=15, cluster=9, every=0):
        bwd = fwd if bwd is None else bwd
        args = [available, cluster, every, len(fwd), *fwd, *bwd]
        r = subprocess.run([out], input=" ".join(str(int(a)) for a in args), text=True,
                           capture_output=True, timeout=60)
        assert r.returncode == 0, r.stdout + r.stderr
        w, *s = r.stdout.split()
        return float(w), tuple(int(v) for v in s)

    return run


def lattice(N):
    """level widths of the N-cell cube in lattice order (6 N levels)"""
    a = np.arange(N + 1)
    d = (a[:, None, None] + 2 * a[None, :, None] + 3 * a[None, None, :]).ravel()
    return np.bincount(d)


@pytest.mark.parametrize("N,want", [(4, (1, 8, 8)), (8, (1, 8, 8)), (16, (1, 12, 10)),
                                    (20, (5, 16, 12)), (32, (12, 16, 14)), (48, (15, 24, 16)),
                                    (64, (15, 32, 16))])
def test_lattice_cubes(shape, N, want):
    assert shape(lattice(N))[1] == want


def test_the_typical_node_decides(shape):
    """a few wide levels among many narrow ones: the mean over levels is that
    of a small mesh, but most nodes sit in wide ones"""
    widths = [5] * 900 + [400] * 100
    w, s = shape(widths)
    assert abs(w - (900 * 25 + 100 * 160000) / sum(widths)) < 1e-6
    assert s == (15, 16, 14) and shape([45] * 1000)[1] == (1, 12, 10)


def test_the_wider_direction_decides(shape):
    narrow, wide = [20] * 100, [200] * 10 + [0] * 90
    assert shape(narrow)[1] == (1, 8, 8)
    assert shape(narrow, wide)[1] == shape(wide, narrow)[1] == shape([200] * 10)[1] == (9, 16, 12)


def test_caps(shape):
    assert shape([1])[1] == (1, 8, 8)
    assert shape([500] * 50, available=3)[1][0] == 3
    assert shape([100000] * 10)[1] == (15, 32, 16)
    # a plan on few clusters did not fit: all of them, enough warps each
    assert shape([25] * 800, every=1)[1] == (15, 16, 12)
