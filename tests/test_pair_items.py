"""The pair kernels at the edges of their work items: 1 to 300 particles per cell (lane groups of 8, 4, 2 and 1, chunks
of 32 particles and one more, one to seventeen stages of candidates, sweeps over more hits than the list queue
holds), the parts of a cell that a few crowded cells are split into, and images in nearly every cell.  Tolerances
as in test_gpu_parity."""
import numpy as np
import pytest

from test_gpu_parity import TOL, assert_same_pairs

pytestmark = pytest.mark.gpu

BOXES = {"ortho3": (3, [3.3, 3.4, 3.5]), "tri3": (3, [[3.3, 0.4, 0.2], [0.0, 3.4, 0.3], [0.0, 0.0, 3.5]]), "none3": (3, None),
         "ortho2": (2, [3.3, 3.4]), "tri2": (2, [[3.3, 0.4], [0.0, 3.4]]), "none2": (2, None)}


def points(dim, per_cell, seed, dtype):
    """per_cell points in each cell of a 3 x 3 (x 3) grid over a box of side 3.3."""
    rng = np.random.default_rng(seed)
    corner = np.stack(np.meshgrid(*[np.arange(3) * 1.1] * dim, indexing="ij"), -1).reshape(-1, 1, dim)
    x = (corner + 1.1 * rng.random((corner.shape[0], per_cell, dim))).reshape(-1, dim)
    return rng.permutation(x).astype(dtype)


@pytest.mark.parametrize("box", list(BOXES))
@pytest.mark.parametrize("per_cell", [1, 4, 5, 8, 9, 16, 17, 32, 33, 65, 300])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_self_pairs(clm, orc, per_cell, box, dtype):
    dim, uc = BOXES[box]
    kind = {"o": "ortho", "t": "tri", "n": "nonperiodic"}[box[0]]
    x = points(dim, per_cell, 3 * per_cell + dim, dtype)
    kw = dict(dim=dim, kind=kind, unitcell=uc, cutoff=1.0, dtype=dtype, nthreads=4)
    ref = orc.run("nl", x, **kw)
    for prec in ("exact", "split"):
        s = clm.ParticleSystem(xpositions=x, unitcell=uc, cutoff=1.0, dtype=dtype, precision=prec)
        exact = prec == "exact" or dtype == np.float32
        assert_same_pairs(orc, clm.pairwise(clm.NeighborList(), s), ref, exact_d=exact, d_rtol=1e-6, d_atol=2e-6)
        assert clm.pairwise(clm.Count(), s) == len(ref["i"])
        tol = TOL[dtype] if prec == "exact" else 1e-5
        r = orc.run("soft_forces", x, **kw)
        ef = clm.pairwise(clm.SoftForces(), s)
        assert abs(ef.energy - r["scalar"]) <= tol * abs(r["scalar"])
        scale = np.abs(r["forces_x"]).max() if len(ref["i"]) else 1e-300
        ftol = tol if prec == "exact" else 1e-4
        assert np.abs(np.asarray(ef.forces, np.float64) - r["forces_x"]).max() <= ftol * scale
        e = clm.pairwise(clm.SoftEnergy(), s)
        assert abs(e - r["scalar"]) <= tol * abs(r["scalar"])
        s.close()


@pytest.mark.parametrize("box", list(BOXES))
@pytest.mark.parametrize("per_cell", [1, 8, 17, 33, 200])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_cross_pairs(clm, orc, per_cell, box, dtype):
    dim, uc = BOXES[box]
    kind = {"o": "ortho", "t": "tri", "n": "nonperiodic"}[box[0]]
    x, y = points(dim, per_cell, per_cell, dtype), points(dim, (per_cell + 1) // 2, 7 + per_cell, dtype)
    kw = dict(dim=dim, kind=kind, unitcell=uc, cutoff=1.0, dtype=dtype, nthreads=4)
    ref = orc.run("nl", x, y, **kw)
    s = clm.ParticleSystem(xpositions=x, ypositions=y, unitcell=uc, cutoff=1.0, dtype=dtype)
    assert_same_pairs(orc, clm.pairwise(clm.NeighborList(), s), ref, cross=True)
    i, j, d = clm.pairwise(clm.MinimumDistance(), s)
    k = int(np.argmin(ref["d"]))
    assert (i, j) == (ref["i"][k], ref["j"][k]) and d == ref["d"][k]
    vx, vy = np.random.default_rng(1).normal(size=x.shape).astype(dtype), np.random.default_rng(2).normal(size=y.shape).astype(dtype)
    bins = np.linspace(0.0, 1.0, 21)
    hc, _ = clm.pairwise(clm.RadialHistogram(bins, vx, vy), s)
    np.testing.assert_array_equal(hc, orc.run("rhist", x, y, bins=bins, vel_x=vx, vel_y=vy, **kw)["hist_count"])
    s.close()
