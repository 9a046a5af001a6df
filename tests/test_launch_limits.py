"""Host side of the kernel launches against a fake CUDA runtime
(tests/cpp/fake_cudart.hpp): no device is needed, and refused launches cost
nothing.  The library's own sources are compiled as they are; only the
runtime under them is replaced."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "atlas-flexmesh_b200", "csrc")
CPP = os.path.join(ROOT, "tests", "cpp")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    """exe(check, sources): builds tests/cpp/<check>.cu with the library's
    sources and the fake runtime (PTX only: nothing of it is ever run)"""
    import sys

    sys.path.insert(0, os.path.join(ROOT, "atlas-flexmesh_b200"))
    import build as B

    out = tmp_path_factory.mktemp("fake")

    def one(check, sources):
        flags = ["-gencode", "arch=compute_100a,code=compute_100a", "-O1", "-std=c++17", "-ccbin",
                 B.host_cxx(), "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-I", CPP]
        files = [os.path.join(CPP, check + ".cu"), os.path.join(CPP, "fake_cudart.cpp")]
        files += [os.path.join(CSRC, s) for s in sources]
        objs = {f: str(out / (os.path.basename(f) + ".o")) for f in files}
        jobs = [subprocess.Popen([B.nvcc(), *flags, "-c", "-o", o, f])
                for f, o in objs.items() if not os.path.exists(o)]
        assert [j.wait(timeout=600) for j in jobs] == [0] * len(jobs)
        prog = str(out / check)
        # what the check does not reach stays unresolved
        subprocess.run([B.host_cxx(), "-o", prog, *objs.values(), "-Wl,--unresolved-symbols=ignore-all",
                        "-lpthread"], check=True, timeout=300)
        return prog

    return one


def run(prog, *args):
    r = subprocess.run([prog, *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_one_shared_memory_limit_per_kernel(exe):
    run(exe("launch_limits_check", ["fm_spmv.cu", "fm_trsv_small.cu"]))


LIB = ["fm_api.cu", "fm_kernels.cu", "fm_nodes.cu", "fm_trsv.cu", "fm_trsv_push.cu",
       "fm_trsv_small.cu", "fm_spmv.cu", "fm_adjoint.cu", "fm_states.cu", "fm_meshsetup.cu",
       "fm_setup.cpp", "fm_checkpoint.cpp"]


def test_refused_launches_are_reported(exe):
    run(exe("launch_failures_check", LIB))


def test_csr_routes(exe):
    run(exe("csr_routes_check", LIB))
