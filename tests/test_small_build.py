"""The one-launch build of small sets (k_build_small): the cell list must equal the oracle's copy by copy at the edges
of its warps, blocks and cell ranges, on repeated builds (its two sets of counters alternate), when the box or the
number of cells changes between builds, and when a cell has more copies than a bucket holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOXES = {"ortho": [9.0, 10.0, 11.0], "tri": [[9.0, 1.0, 0.5], [0.0, 10.0, 1.5], [0.0, 0.0, 11.0]], "nonperiodic": None,
         "ortho2": [9.0, 10.0], "tri2": [[9.0, 1.5], [0.0, 10.0]]}


def check(clm, orc, s, x, dim, kind, uc, cut, dtype):
    cl = s.fetch_celllist(0)
    oc = orc.celllist(x, dim=dim, kind=kind, unitcell=uc, cutoff=cut, dtype=dtype)
    for k in ("cell", "index", "real"):
        np.testing.assert_array_equal(cl[k], oc[k])
    np.testing.assert_array_equal(cl["coords"].astype(np.float64), oc["coords"])


@pytest.mark.parametrize("box", list(BOXES))
@pytest.mark.parametrize("n", [1, 31, 32, 33, 4863, 4865, 40000])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_cell_list_copy_by_copy(clm, orc, n, box, dtype):
    uc = BOXES[box]
    dim, kind = (2, box[:-1]) if box[-1] == "2" else (3, box)
    rng = np.random.default_rng(n)
    x = (rng.random((n, dim)) * 24.0 - 7.0).astype(dtype)
    s = clm.ParticleSystem(xpositions=x, unitcell=uc, cutoff=1.1, dtype=dtype)
    for cut in (1.1, 1.1, 0.8, 1.1):
        s.update(xpositions=x, cutoff=cut)
        s.build()
        check(clm, orc, s, x, dim, kind, uc, cut, dtype)
        x = (x + dtype(0.37)).astype(dtype)
    s.close()


@pytest.mark.parametrize("blob", [127, 128, 129, 900, 2500])
def test_full_buckets(clm, orc, blob):
    """blob particles in one cell of a box whose other cells hold about three: 128 fit a bucket, 129 make the set fall
    back to the counting build, 2500 further to radix."""
    rng = np.random.default_rng(blob)
    x = np.concatenate([20.0 * rng.random((20000, 3)), 10.3 + 0.2 * rng.random((blob, 3))])
    x = x[(np.abs(x - 10.5).max(1) > 0.6) | (np.arange(len(x)) >= 20000)]
    s = clm.ParticleSystem(xpositions=x, unitcell=[20.0] * 3, cutoff=1.0)
    ref = orc.run("count", x, unitcell=[20.0] * 3, cutoff=1.0)["count"]
    for _ in range(3):
        s.update(xpositions=x)
        assert clm.pairwise(clm.Count(), s) == ref
        check(clm, orc, s, x, 3, "ortho", [20.0] * 3, 1.0, np.float64)
    s.close()
