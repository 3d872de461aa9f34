"""What a particle set remembers from one build to the next (clm_build_state.hpp): the alternating counters of the
small build start clear after every mixture of launches, dropped and failed ones, and a list that a build with an
error left is never used by a later call.  Runs on the CPU."""
import ctypes as C
import itertools
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = str(tmp_path_factory.mktemp("state") / "libstate.so")
    inc = next((os.path.join(c, "include") for c in (os.environ.get("CUDA_HOME", ""), "/usr/local/cuda")
                if c and os.path.exists(os.path.join(c, "include", "cuda_runtime.h"))), None)
    if inc is None:
        pytest.skip("no CUDA headers")
    r = subprocess.run([cxx, "-O1", "-std=c++17", "-fPIC", "-shared", "-I", inc, "-I", os.path.join(ROOT, "celllistmap.jl_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "build_state_probe.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(out)


def test_small_counters_start_clear(probe):
    """Every sequence of six steps (launched, dropped before the launch, refused, other grid, new memory)."""
    for script in itertools.product(range(5), repeat=6):
        a = (C.c_int * 6)(*script)
        assert probe.small_counters_probe(a, 6) == -1, script


NAN, RANGE, COPIES, SCAN = 1, 2, 4, 16


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("errw,status", [(0, 0), (NAN, 3), (RANGE, 12), (SCAN, 12), (SCAN | RANGE, 12), (NAN | SCAN, 3),
                                         (SCAN | COPIES, 12)])
def test_an_error_leaves_no_list_in_use(probe, kind, errw, status):
    out = (C.c_int * 8)()
    probe.check_probe(kind, errw, 900, 20, out)
    assert out[0] == status
    for dirty, pending, cleared in (out[2:5], out[5:8]):
        assert dirty == (errw != 0)             # built again by the next call
        assert cleared == bool(errw & SCAN)     # and not on words that a block left half written
