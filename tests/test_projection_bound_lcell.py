"""The bound below which a Float64 pair skips the projection filter (test_projection_bound), for lcell 4 to 12.  Runs on
the CPU."""
import ctypes as C

import numpy as np
import pytest

from tests.test_projection_bound import CASES, KINDS, probe  # noqa: F401


@pytest.mark.parametrize("lcell", [4, 5, 7, 12])
@pytest.mark.parametrize("case", [c for c in CASES if max(np.ravel(c[2])) < 1.0e3], ids=lambda c: f"{c[0]}d-{c[1]}-{c[4]}")
def test_large_lcell(probe, case, lcell):  # noqa: F811
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
