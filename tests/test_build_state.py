"""What a particle set remembers from one build to the next (clm_build_state.hpp): the alternating counters of the
one-launch build start clear after every mixture of launches, dropped and failed ones.  Runs on the CPU."""
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
    r = subprocess.run([cxx, "-O1", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(ROOT, "celllistmap.jl_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "build_state_probe.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(out)


def test_small_counters_start_clear(probe):
    """Every sequence of six steps (launched, dropped before the launch, refused, other grid, new memory)."""
    for script in itertools.product(range(5), repeat=6):
        a = (C.c_int * 6)(*script)
        assert probe.small_counters_probe(a, 6) == -1, script
