"""Hits found by one lane and evaluated by the others: a stage's hits are shared out evenly over the warp, so with one
particle of a chunk near hundreds of candidates and 31 near none every lane reads a mask that another lane wrote, and
the list's queue of a dense cell is reduced in place over many passes.  Every list, count and minimum is exact."""
import numpy as np
import pytest

from test_gpu_parity import TOL, assert_same_pairs

pytestmark = pytest.mark.gpu


def points(kind, rng, dtype):
    if kind == "one_lane":  # the last of 32 particles of a cell, beside a cluster in the next cell
        far = np.array([1.05, 1.05, 1.05]) + 0.02 * rng.random((31, 3))
        near = np.array([[1.95, 1.5, 1.5]])
        cluster = np.array([2.2, 1.4, 1.4]) + 0.2 * rng.random((250, 3))
        x = np.concatenate([far, near, cluster])
    else:  # every candidate of every particle is a hit
        x = 1.5 + 0.4 * rng.random((700, 3))
    return x.astype(dtype)


@pytest.mark.parametrize("kind", ["one_lane", "all_hits"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_hits_of_other_lanes(clm, orc, kind, dtype):
    kw = dict(unitcell=[6.0, 6.0, 6.0], cutoff=1.0, dtype=dtype)
    s = None
    for seed in range(20):
        x = points(kind, np.random.default_rng(seed), dtype)
        if s is None:
            s = clm.ParticleSystem(xpositions=x, **kw)
        else:
            s.update(xpositions=x)
        ref = orc.run("nl", x, **kw)
        assert_same_pairs(orc, clm.pairwise(clm.NeighborList(), s), ref)
        assert clm.pairwise(clm.Count(), s) == len(ref["i"])
        r = orc.run("soft_forces", x, **kw)
        ef = clm.pairwise(clm.SoftForces(), s)
        assert abs(ef.energy - r["scalar"]) <= TOL[dtype] * abs(r["scalar"])
        assert np.abs(np.asarray(ef.forces, np.float64) - r["forces_x"]).max() <= TOL[dtype] * np.abs(r["forces_x"]).max()
        i, j, d = clm.pairwise(clm.MinimumDistance(), s)
        k = int(np.argmin(ref["d"]))
        assert {i, j} == {ref["i"][k], ref["j"][k]} and d == ref["d"][k]
    s.close()
