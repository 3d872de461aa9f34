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


def crowding(probe, kind, most):
    n = len(kind)
    out = (C.c_int * (10 * n))()
    probe.crowding_probe(n, (C.c_int * (2 * n))(*sum(kind, [])), (C.c_int * (2 * n))(*sum(most, [])), out)
    return [(tuple(out[10 * k:10 * k + 5]), tuple(out[10 * k + 5:10 * k + 10])) for k in range(n)]


CLEAN = (0, 0, 0, 0, 2)


@pytest.mark.parametrize("other", [0, 1, 2])
@pytest.mark.parametrize("first", [0, 1])
def test_an_overflow_is_one_sets_own(probe, other, first):
    """The other set of the handle, whose cells fit, is not built again and keeps its builds."""
    kind, most = [[1, other]], [[129, 20]]
    if first:
        kind, most = [[other, 1]], [[20, 129]]
    st = crowding(probe, kind, most)[0]
    assert st[first] == (1, 0, 168, 1, 2) and st[1 - first] == CLEAN


def test_one_crowded_step_is_forgotten(probe):
    """129 copies leave the small build for buckets of 168, 300 the buckets for the counting build; when the fullest
    cell leaves a quarter free the builds are taken again, and not before."""
    kind = [[1, 3], [2, 3], [2, 3], [2, 3], [0, 3], [0, 3], [0, 3], [2, 3], [1, 3]]
    most = [[129, 0], [129, 0], [300, 0], [300, 0], [300, 0], [193, 0], [192, 0], [96, 0], [20, 0]]
    got = [a for a, _ in crowding(probe, kind, most)]
    assert [g[0] for g in got] == [1, 1, 1, 1, 1, 1, 1, 0, 0]       # small_off
    assert [g[1] for g in got] == [0, 0, 1, 1, 1, 1, 0, 0, 0]       # bucket_off
    assert got[0][2] == 168 and got[6][2] == 240 and got[7][2] == 120
    assert all(g[4] == 2 for g in got)
