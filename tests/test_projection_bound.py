"""The pair kernel keeps a Float64 pair of d2 <= proj_lo without the reference's projection filter
(vicinal_cells.jl:4-75): the filter must keep every such pair, also where it is closest to rejecting it (particles on
cell faces, separations along the line of two cell centres, distances a few units below the bound), for small and large
boxes, lcell 1 to 3 and boxes far from the origin.  Runs on the CPU."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from tests.conftest import ROOT

KINDS = {"ortho": 0, "tri": 1, "nonperiodic": 2}
CASES = [
    (3, "ortho", [20.0, 21.0, 22.0], None, 1.1),
    (3, "ortho", [1000.0, 1100.0, 9.0], None, 1.0),
    (3, "ortho", [1.0e5, 3.0, 3.0], None, 1.0),
    (3, "tri", [[20.0, 4.0, 2.0], [0.0, 20.0, 3.0], [0.0, 0.0, 20.0]], None, 1.3),
    (3, "tri", [[14.0, 9.0, -6.0], [1.0, 15.0, 7.0], [-2.0, 3.0, 16.0]], None, 0.7),
    (3, "nonperiodic", [20.0, 21.0, 22.0], [1.0e6, -3.0e4, 0.0], 1.1),
    (3, "nonperiodic", [20.0, 21.0, 22.0], [1.0e9, 0.0, 0.0], 1.1),
    (2, "ortho", [30.0, 25.0], None, 0.1),
    (2, "tri", [[30.0, 14.0], [0.0, 25.0]], None, 0.9),
]


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    inc = next((os.path.join(c, "include") for c in (os.environ.get("CUDA_HOME", ""), "/usr/local/cuda")
                if c and os.path.exists(os.path.join(c, "include", "cuda_runtime.h"))), None)
    if cxx is None or inc is None:
        pytest.skip("no C++ compiler or CUDA headers")
    out = str(tmp_path_factory.mktemp("proj") / "libproj_probe.so")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-fno-fast-math", "-I", inc, "-I",
                        os.path.join(ROOT, "celllistmap.jl_gb300", "csrc"), os.path.join(ROOT, "tests", "proj_probe.cpp"),
                        "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(out)


@pytest.mark.parametrize("lcell", [1, 2, 3])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}d-{c[1]}-{c[4]}")
def test_the_filter_keeps_every_pair_below_the_bound(probe, case, lcell):
    dim, kind, uc, origin, cutoff = case
    uc = np.asarray(uc, np.float64)
    M = np.ascontiguousarray((np.diag(uc) if uc.ndim == 1 else uc).flatten(order="F"))
    o = None if origin is None else np.asarray(origin, np.float64)
    out = np.zeros(4, np.int64)
    st = probe.proj_probe(dim, KINDS[kind], M.ctypes.data_as(C.c_void_p),
                          None if o is None else o.ctypes.data_as(C.c_void_p), C.c_double(cutoff), lcell, 400000,
                          out.ctypes.data_as(C.c_void_p))
    assert st == 0
    tested, above, rejected, wider = out
    assert tested > 1000 and rejected == 0
    assert not wider or above > 1000  # the pairs that the bound takes from the filter were among them
