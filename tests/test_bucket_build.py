"""The build of large sets and of batches through a bucket per cell (k_wrap_place, k_cell_scan, k_bucket_gather): the
cell list must equal the oracle's copy by copy at the edges of its blocks of particles and of cells, from sparse to full
buckets, on repeated builds (the scan words are cleared by the build before), and when a cell has more copies than its
bucket holds.  The list is exact, so there is no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOXES = {"ortho": [20.0, 21.0, 22.0], "tri": [[20.0, 2.0, 1.0], [0.0, 21.0, 3.0], [0.0, 0.0, 22.0]], "nonperiodic": None,
         "ortho2": [200.0, 210.0], "tri2": [[200.0, 30.0], [0.0, 210.0]]}


def check(clm, orc, s, x, dim, kind, uc, cut, dtype):
    cl = s.fetch_celllist(0)
    oc = orc.celllist(x, dim=dim, kind=kind, unitcell=uc, cutoff=cut, dtype=dtype)
    for k in ("cell", "index", "real"):
        np.testing.assert_array_equal(cl[k], oc[k])
    np.testing.assert_array_equal(cl["coords"].astype(np.float64), oc["coords"])


@pytest.mark.parametrize("box", list(BOXES))
@pytest.mark.parametrize("n", [65537, 65792, 70001])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_cell_list_copy_by_copy(clm, orc, n, box, dtype):
    uc = BOXES[box]
    dim, kind = (2, box[:-1]) if box[-1] == "2" else (3, box)
    rng = np.random.default_rng(n)
    side = 1.0 if dim == 3 else 9.5
    x = (rng.random((n, dim)) * (uc[-1] if kind == "ortho" else 40.0) * 1.3 - 7.0).astype(dtype)
    if kind != "ortho":
        x = (rng.random((n, dim)) * 21.0 * side).astype(dtype)
    s = clm.ParticleSystem(xpositions=x, unitcell=uc, cutoff=1.1, dtype=dtype)
    for cut in (1.1, 1.1, 0.6, 1.9) if dim == 3 else (1.1, 1.1, 2.0, 6.0):
        s.update(xpositions=x, cutoff=cut)
        s.build()
        check(clm, orc, s, x, dim, kind, uc, cut, dtype)
        x = (x + dtype(0.37)).astype(dtype)
    s.close()


@pytest.mark.parametrize("blob", [20, 70, 100, 130, 900, 2500])
def test_full_buckets(clm, orc, blob):
    """blob particles in one cell of a box whose other cells hold about six: up to two hundred the buckets grow, more
    make the set fall back to the counting build and then to radix."""
    rng = np.random.default_rng(blob)
    x = np.concatenate([23.0 * rng.random((70000, 3)), 10.3 + 0.2 * rng.random((blob, 3))])
    s = clm.ParticleSystem(xpositions=x, unitcell=[23.0] * 3, cutoff=1.0)
    ref = orc.run("count", x, unitcell=[23.0] * 3, cutoff=1.0)["count"]
    for _ in range(3):
        s.update(xpositions=x)
        assert clm.pairwise(clm.Count(), s) == ref
        check(clm, orc, s, x, 3, "ortho", [23.0] * 3, 1.0, np.float64)
    s.close()


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("blob", [0, 60, 300])
def test_batch(clm, orc, blob, graph):
    """Systems of different densities in one batch (one of them empty, one with a blob): counts of each against the
    oracle, over repeated steps with and without a recorded step."""
    rng = np.random.default_rng(7)
    cut, L = 1.0, np.array([9.0, 2.5, 6.0, 4.0])
    xs = [l * rng.random((m, 3)) for l, m in zip(L, (3000, 200, 0, 257))]
    if blob:
        xs[0][:blob] = 4.2 + 0.2 * rng.random((blob, 3))
    b = clm.BatchedSystems(positions=xs, unitcells=[[l] * 3 for l in L], cutoff=cut, graph=graph)
    for _ in range(3):
        xs = [x + 0.21 for x in xs]
        b.update(positions=np.concatenate(xs))
        ref = [orc.run("count", x, unitcell=[l] * 3, cutoff=cut)["count"] if len(x) else 0 for x, l in zip(xs, L)]
        assert b.run(clm.Count())[0].tolist() == ref
