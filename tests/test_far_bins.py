"""The exact radial histogram takes a pair's bin from the FP32 distance of the cell offsets unless an edge lies within
that distance's error: the error must stay within the bound the kernel is given (offset_distance_error), and every bin
that is not decided again must be the one of the Float64 distance, near the origin and far from it.  Runs on the CPU."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from tests.conftest import ROOT


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    inc = next((os.path.join(c, "include") for c in (os.environ.get("CUDA_HOME", ""), "/usr/local/cuda")
                if c and os.path.exists(os.path.join(c, "include", "cuda_runtime.h"))), None)
    if cxx is None or inc is None:
        pytest.skip("no C++ compiler or CUDA headers")
    out = str(tmp_path_factory.mktemp("far") / "libfar_probe.so")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-fno-fast-math", "-I", inc, "-I",
                        os.path.join(ROOT, "celllistmap.jl_gb300", "csrc"), os.path.join(ROOT, "tests", "far_probe.cpp"),
                        "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(out)


@pytest.mark.parametrize("dim,side,cutoff", [(3, [20.0, 21.0, 22.0], 1.1), (3, [0.8, 0.9, 5.0], 0.01),
                                             (2, [300.0, 250.0], 1.0)])
@pytest.mark.parametrize("lcell", [1, 3])
@pytest.mark.parametrize("origin", [0.0, 1.0e3, 1.0e6, 1.0e8, 1.0e9, 1.0e10])
def test_bins_from_the_offsets(probe, origin, lcell, dim, side, cutoff):
    if origin / cutoff > 1e10:
        pytest.skip("the coordinates resolve the cutoff to less than the band around it")
    out = np.zeros(4, np.int64)
    sd = np.asarray(side, np.float64)
    st = probe.far_probe(dim, sd.ctypes.data_as(C.c_void_p), C.c_double(origin), C.c_double(cutoff), lcell, 200000, 50,
                         out.ctypes.data_as(C.c_void_p))
    assert st == 0
    tested, beyond, wrong, again = out
    assert tested > 100000 and beyond == 0 and wrong == 0
    if origin <= 1e3:
        assert again < tested  # most bins stand as they are
