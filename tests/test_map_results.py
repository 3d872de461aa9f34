"""The kernel that ends a map (k_finish: partials reduced, histogram and adjoint columns summed, forces converted),
at the edges of its blocks of 256 threads and of its warp-per-column sums.  Tolerances as in test_gpu_parity."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (255, 257), (256, 1), (513, 256), (1, 0), (300, 0)])
@pytest.mark.parametrize("dtype,tol", [(np.float64, 1e-12), (np.float32, 1e-5)])
def test_forces_of_both_sets(clm, orc, nx, ny, dtype, tol):
    rng = np.random.default_rng(nx + 7 * ny)
    x = (rng.random((nx, 3)) * 9.0).astype(dtype)
    y = (rng.random((ny, 3)) * 9.0).astype(dtype) if ny else None
    M = [[9.0, 1.0, 0.5], [0.0, 9.0, 1.5], [0.0, 0.0, 9.0]]
    s = clm.ParticleSystem(xpositions=x, ypositions=y, unitcell=M, cutoff=4.0, dtype=dtype)
    r = orc.run("soft_forces", x, y, kind="tri", unitcell=M, cutoff=4.0, dtype=dtype)
    ef = clm.pairwise(clm.SoftForces(), s)
    assert abs(ef.energy - r["scalar"]) <= tol * abs(r["scalar"])
    for got, ref in ((ef.forces, r["forces_x"]),) + (((ef.forces_y, r["forces_y"]),) if ny else ()):
        assert np.abs(np.asarray(got, np.float64) - ref).max() <= tol * max(np.abs(ref).max(), 1e-300)
    i, j, d = clm.pairwise(clm.MinimumDistance(), s)
    nl = orc.run("nl", x, y, kind="tri", unitcell=M, cutoff=4.0, dtype=dtype)
    if len(nl["d"]) == 0:
        assert (i, j) == (-1, -1)
    else:
        k = int(np.argmin(nl["d"]))
        assert (i, j) == (nl["i"][k], nl["j"][k]) and d == nl["d"][k]
    s.close()


@pytest.mark.parametrize("nbins", [1, 7, 8, 9, 50, 256])
def test_histogram_columns(clm, orc, nbins):
    rng = np.random.default_rng(nbins)
    x, y = rng.random((700, 3)) * 10.0, rng.random((500, 3)) * 10.0
    vx, vy = rng.normal(0.0, 300.0, x.shape), rng.normal(0.0, 300.0, y.shape)
    bins = np.linspace(0.2, 4.0, nbins + 1)
    s = clm.ParticleSystem(xpositions=x, ypositions=y, unitcell=[10.0] * 3, cutoff=4.0)
    hc, hs = clm.pairwise(clm.RadialHistogram(bins, vx, vy), s)
    r = orc.run("rhist", x, y, unitcell=[10.0] * 3, cutoff=4.0, vel_x=vx, vel_y=vy, bins=bins)
    np.testing.assert_array_equal(hc, r["hist_count"])
    assert np.abs(hs - r["hist_sum"]).max() <= 1e-10 * np.abs(r["hist_sum"]).max()
    s.close()
