"""Builds of the two sets of an x-y system: the limits of both in one launch (k_limits) and, for small sets, both cell
lists in one launch of k_build_small, whose blocks are split between the sets.  Pair lists against the oracle at the
edges of blocks and of that split, with one set far larger than the other, one empty, or one built by another build."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 5000), (5000, 3), (255, 257), (1501, 4507), (40000, 65536), (300, 70000), (0, 400), (700, 0)]


def pairs(clm, s):
    i, j, d = clm.pairwise(clm.NeighborList(), s)
    o = np.lexsort((j, i))
    return i[o], j[o], d[o]


@pytest.mark.parametrize("kind", ["nonperiodic", "ortho"])
@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_cross_pairs(clm, orc, nx, ny, kind, dtype):
    rng = np.random.default_rng(nx + 7 * ny)
    side = max(4.0, (max(nx, ny) / 2.0) ** (1.0 / 3.0))
    uc = None if kind == "nonperiodic" else [side] * 3
    x = (side * rng.random((nx, 3)) - 1.0).astype(dtype)
    y = (side * rng.random((ny, 3)) - 1.3).astype(dtype)
    s = clm.ParticleSystem(xpositions=x, ypositions=y, unitcell=uc, cutoff=0.6, dtype=dtype)
    for step in range(3):
        ref = orc.run("nl", x, y=y, kind=kind, unitcell=uc, cutoff=0.6, dtype=dtype)
        o = np.lexsort((ref["j"], ref["i"]))
        i, j, d = pairs(clm, s)
        np.testing.assert_array_equal(i, ref["i"][o])
        np.testing.assert_array_equal(j, ref["j"][o])
        # one rounding of d2 and of the root, in the handle's type
        np.testing.assert_allclose(d, ref["d"][o], rtol=4 * np.finfo(dtype).eps)
        if step == 0:  # both sets move
            x, y = (x + dtype(0.3)).astype(dtype), (y * dtype(1.1)).astype(dtype)
            s.update(xpositions=x, ypositions=y)
        elif nx:       # one set moves
            x = (x - dtype(0.2)).astype(dtype)
            s.update(xpositions=x)
    s.close()
