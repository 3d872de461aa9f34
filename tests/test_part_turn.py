"""Cells in parts whose number shares factors with the number of warps (the parts of a cell are turned from wave to
wave): every part of every cell is mapped once, so counts and lists are exact.  One to five waves of items, and the
specialised split forces of the soft potential."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rc", [(1003, 5.0), (20001, 8.0), (60000, 7.0), (100003, 8.0), (100003, 4.0)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_every_part_once(clm, orc, n, rc, dtype):
    side = (n / 0.1) ** (1.0 / 3.0)
    x = (side * np.random.default_rng(n).random((n, 3))).astype(dtype)
    kw = dict(unitcell=[side] * 3, cutoff=rc, dtype=dtype)
    ref = orc.run("nl", x, nthreads=4, **kw)
    s = clm.ParticleSystem(xpositions=x, **kw)
    assert clm.pairwise(clm.Count(), s) == len(ref["i"])
    a = orc.canonical_pairs(*clm.pairwise(clm.NeighborList(), s))
    b = orc.canonical_pairs(ref["i"], ref["j"], ref["d"])
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[1], b[1])
    e = clm.pairwise(clm.SoftEnergy(), s)
    assert e == clm.pairwise(clm.SoftEnergy(), s)  # summed in a fixed order
    s.close()


@pytest.mark.parametrize("n,rc", [(1003, 5.0), (20001, 8.0)])
@pytest.mark.parametrize("kind", ["ortho", "tri", "cross", "2d"])
def test_split_soft_forces(clm, orc, n, rc, kind):
    dim = 2 if kind == "2d" else 3
    side = (n / 0.1) ** (1.0 / dim)
    M = np.eye(dim) * side
    if kind == "tri":
        M[0, 1] = 0.2 * side
    uc = M if kind == "tri" else [side] * dim
    rng = np.random.default_rng(n)
    x = rng.random((n, dim)) @ M.T
    y = rng.random((n // 2, dim)) @ M.T if kind == "cross" else None
    kw = dict(unitcell=uc, cutoff=rc)
    r = orc.run("soft_forces", x, y, dim=dim, kind="tri" if kind == "tri" else "ortho", nthreads=4, **kw)
    s = clm.ParticleSystem(xpositions=x, ypositions=y, precision="split", **kw)
    ef = clm.pairwise(clm.SoftForces(), s)
    assert abs(ef.energy - r["scalar"]) <= 1e-5 * abs(r["scalar"])  # the tolerances of test_gpu_parity
    for got, want in ((ef.forces, r["forces_x"]),) + (((ef.forces_y, r["forces_y"]),) if kind == "cross" else ()):
        assert np.abs(np.asarray(got) - want).max() <= 1e-4 * np.abs(want).max()
    s.close()
