"""A step of a small system runs beside a kernel of another stream that holds most of the multiprocessors: no launch of
the step needs more of the device at once than is left.  The other kernel holds 140 of 152 multiprocessors for 200 ms and ends by itself; a
step takes a tenth of a millisecond."""
import ctypes as C
import os
import subprocess
import time

import numpy as np
import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hold(clm, tmp_path_factory):
    out = str(tmp_path_factory.mktemp("hold") / "libhold.so")
    r = subprocess.run([clm.build_lib.nvcc(), "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_103a,code=sm_103a",
                        os.path.join(ROOT, "tests", "hold_kernel.cu"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(out)
    lib.hold.argtypes = [C.c_int, C.c_longlong, C.c_void_p]
    return lib


@pytest.mark.parametrize("nx,ny", [(1000, 0), (40000, 0), (4000, 3000)])
def test_a_step_beside_a_long_kernel(clm, hold, nx, ny):
    import torch

    rng = np.random.default_rng(nx)
    p = {"xpositions": 20.0 * rng.random((nx, 3))}
    if ny:
        p["ypositions"] = 20.0 * rng.random((ny, 3))
    s = clm.ParticleSystem(**p, unitcell=[20.0] * 3, cutoff=1.0)
    count = clm.pairwise(clm.Count(), s)
    other, ended = torch.cuda.Stream(), torch.cuda.Event()
    assert hold.hold(1, 1000, other.cuda_stream) == 0  # loads the module
    torch.cuda.synchronize()
    assert hold.hold(140, 200_000_000, other.cuda_stream) == 0
    ended.record(other)
    time.sleep(0.02)  # it has begun
    for _ in range(3):
        s.update(**p)
        assert clm.pairwise(clm.Count(), s) == count
    beside = not ended.query()
    torch.cuda.synchronize()
    s.close()
    assert beside, "the step waited for the other stream's kernel"
