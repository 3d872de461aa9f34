"""A small set with a NaN coordinate: its build (k_small_place, k_small_cells) leaves a whole cell list of the other particles, because
the map enqueued behind it runs before the host reads the error.  The call answers with the NaN error, and the steps
after it, on this handle and on another one, equal the oracle."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {np.float64: 1e-12, np.float32: 1e-5}  # the tolerances of test_map_results


def check_forces(clm, orc, s, x, kind, uc, cut, dtype):
    r = orc.run("soft_forces", x, kind=kind, unitcell=uc, cutoff=cut, dtype=dtype)
    ef = clm.pairwise(clm.SoftForces(), s)
    assert abs(ef.energy - r["scalar"]) <= TOL[dtype] * abs(r["scalar"])
    assert np.abs(np.asarray(ef.forces, np.float64) - r["forces_x"]).max() <= TOL[dtype] * np.abs(r["forces_x"]).max()


@pytest.mark.parametrize("kind,uc", [("ortho", [9.0, 10.0, 11.0]), ("nonperiodic", None)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_fewer_particles_with_a_nan(clm, orc, kind, uc, dtype):
    rng = np.random.default_rng(3)
    big = (9.0 * rng.random((60000, 3))).astype(dtype)
    other = (9.0 * rng.random((2000, 3))).astype(dtype)
    s = clm.ParticleSystem(xpositions=big, unitcell=uc, cutoff=0.4, dtype=dtype)
    t = clm.ParticleSystem(xpositions=other, unitcell=uc, cutoff=1.1, dtype=dtype)
    clm.pairwise(clm.SoftForces(), s)
    check_forces(clm, orc, t, other, kind, uc, 1.1, dtype)
    x = (9.0 * rng.random((1000, 3))).astype(dtype)
    for bad in (0, 517, 999):
        y = x.copy()
        y[bad, bad % 3] = np.nan
        s.update(xpositions=y, cutoff=1.1)
        with pytest.raises(Exception, match="NaN"):
            clm.pairwise(clm.SoftForces(), s)
        s.update(xpositions=x)
        check_forces(clm, orc, s, x, kind, uc, 1.1, dtype)
        check_forces(clm, orc, t, other, kind, uc, 1.1, dtype)
    s.close()
    t.close()


def test_first_step_with_a_nan(clm):
    """Through the C ABI, without a build before the map: clm_run builds and maps in one go."""
    A = clm._abi
    L = A.load()
    x = 9.0 * np.random.default_rng(5).random((4000, 3))
    y = x.copy()
    y[77, 1] = np.nan
    f = np.empty_like(x)
    ref = clm.ParticleSystem(xpositions=x, unitcell=[9.0, 10.0, 11.0], cutoff=1.1)
    want = clm.pairwise(clm.SoftForces(), ref)
    h = C.c_void_p()
    assert L.clm_create(1, 3, 1, C.byref(h)) == 0
    M = (C.c_double * 9)(9, 0, 0, 0, 10, 0, 0, 0, 11)
    assert L.clm_set_box(h, M, 0, 1.1, 1) == 0
    p, o = A.OpParams(), A.Outputs()
    o.forces_x = f.ctypes.data
    assert L.clm_set_positions(h, 0, y.ctypes.data, len(y), 0) == 0
    for _ in range(2):
        assert A.STATUS[L.clm_run(h, A.OP["soft_forces"], C.byref(p), C.byref(o))] == "CLM_ERR_NAN"
    assert L.clm_set_positions(h, 0, x.ctypes.data, len(x), 0) == 0
    assert L.clm_run(h, A.OP["soft_forces"], C.byref(p), C.byref(o)) == 0
    assert abs(o.scalar - want.energy) <= TOL[np.float64] * abs(want.energy)
    assert np.abs(f - want.forces).max() <= TOL[np.float64] * np.abs(want.forces).max()
    assert L.clm_destroy(h) == 0
    ref.close()


@pytest.mark.parametrize("bad_set", ["xpositions", "ypositions"])
def test_nan_in_one_of_two_sets(clm, orc, bad_set):
    """Only the set with the NaN gets new positions afterwards: the other one's list is used as it is."""
    rng = np.random.default_rng(9)
    p = {"xpositions": 9.0 * rng.random((3000, 3)), "ypositions": 9.0 * rng.random((1500, 3))}
    bad = {k: v.copy() for k, v in p.items()}
    bad[bad_set][11, 2] = np.nan
    s = clm.ParticleSystem(**p, unitcell=[9.0, 10.0, 11.0], cutoff=1.1)
    s.update(**bad)
    with pytest.raises(Exception, match="NaN"):
        clm.pairwise(clm.NeighborList(), s)
    s.update(**{bad_set: p[bad_set]})
    ref = orc.run("nl", p["xpositions"], y=p["ypositions"], unitcell=[9.0, 10.0, 11.0], cutoff=1.1)
    a = orc.canonical_pairs(*clm.pairwise(clm.NeighborList(), s))
    b = orc.canonical_pairs(ref["i"], ref["j"], ref["d"])
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[1], b[1])
    s.close()
