"""Radial histograms into the caller's device arrays (clm_outputs.out_on_device): written by a call that succeeds, left
alone by one that fails, and refused without both arrays."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["exact", "split"])
@pytest.mark.parametrize("n", [900, 70000])
def test_device_arrays(clm, n, precision):
    import torch

    A = clm._abi
    L = A.load()
    rng = np.random.default_rng(n)
    side = 12.0 if n < 1000 else 40.0
    x, v = side * rng.random((n, 3)), rng.normal(size=(n, 3))
    bins = np.linspace(0.1, 1.0, 14)
    s = clm.ParticleSystem(xpositions=x, unitcell=[side] * 3, cutoff=1.0, precision=precision)
    want = clm.pairwise(clm.RadialHistogram(bins, v), s)
    p, o = A.OpParams(), A.Outputs()
    p.nbins, p.bins, p.vel_x = 13, bins.ctypes.data, v.ctypes.data
    count = torch.full((13,), -7, dtype=torch.int64, device="cuda")
    total = torch.full((13,), -7.0, dtype=torch.float64, device="cuda")
    o.hist_count, o.hist_sum, o.out_on_device = count.data_ptr(), total.data_ptr(), 1
    torch.cuda.synchronize()

    def run():
        st = L.clm_run(s._handle.h, A.OP["rhist"], C.byref(p), C.byref(o))
        torch.cuda.synchronize()
        return A.STATUS[st]

    bad = x.copy()
    bad[n // 2, 1] = np.nan
    assert L.clm_set_positions(s._handle.h, 0, bad.ctypes.data, n, 0) == 0
    assert run() == "CLM_ERR_NAN"
    assert (count == -7).all() and (total == -7.0).all()
    assert L.clm_set_positions(s._handle.h, 0, x.ctypes.data, n, 0) == 0
    assert run() == "CLM_OK"
    np.testing.assert_array_equal(count.cpu().numpy(), want[0])
    np.testing.assert_allclose(total.cpu().numpy(), want[1], rtol=0, atol=1e-10 * np.abs(want[1]).max())
    for a, b in ((0, total.data_ptr()), (count.data_ptr(), 0), (0, 0)):
        o.hist_count, o.hist_sum = a, b
        assert run() == "CLM_ERR_ARG"
    s.close()
