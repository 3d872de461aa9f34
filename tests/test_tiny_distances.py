"""Float64 pair values at distances whose square is subnormal: 1/d, d and their forces are finite down to squared
distances of 1/max(Float64) (the reference's 1/sqrt(d2)), as for any other distance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [0.8e-154, 1.0e-154, 1.4e-154, 1.6e-154, 1.0e-150, 1.0e-10])
def test_values_at_tiny_distances(clm, d):
    x = np.array([[0.0, 0.0, 0.0], [d, 0.0, 0.0], [9.0, 9.0, 9.0]])
    s = clm.ParticleSystem(xpositions=x, unitcell=None, cutoff=1.0)
    r = np.sqrt(d * d)  # d2 has the few bits that a subnormal leaves
    for op, want in ((clm.SumInvD(), 1.0 / r), (clm.SumD(), r), (clm.SoftEnergy(), (1.0 - r) ** 2)):
        got = clm.pairwise(op, s)
        assert abs(got - want) <= 1e-12 * want, (op.op, got, want)
    s.close()


@pytest.mark.parametrize("cross", [False, True])
@pytest.mark.parametrize("d", [0.8e-154, 1.4e-154, 1.0e-150])
def test_forces_and_histogram_at_tiny_distances(clm, d, cross):
    x = np.array([[0.0, 0.0, 0.0], [d, 0.0, 0.0], [9.0, 9.0, 9.0]])
    p = {"xpositions": x}
    if cross:
        p = {"xpositions": x[[0, 2]], "ypositions": x[[1]]}
    s = clm.ParticleSystem(**p, unitcell=None, cutoff=1.0)
    u = (d / np.sqrt(d * d))  # 1 but for the bits that a subnormal d2 lacks
    ef = clm.pairwise(clm.SoftForces(), s)
    assert abs(ef.energy - 1.0) <= 1e-12
    want = np.zeros_like(p["xpositions"])
    want[0, 0] = -2.0 * u
    if cross:
        np.testing.assert_allclose(ef.forces_y, [[2.0 * u, 0.0, 0.0]], rtol=1e-12)
    else:
        want[1, 0] = 2.0 * u
    np.testing.assert_allclose(ef.forces, want, rtol=1e-12)
    v = np.array([[3.0, 1.0, 2.0], [1.0, 5.0, 2.0], [0.0, 0.0, 0.0]])
    vel = (v[[0, 2]], v[[1]]) if cross else (v,)
    for first in (0.0, -0.3, -1.0e-9):
        hc, hs = clm.pairwise(clm.RadialHistogram(np.array([first, 0.5, 1.0]), *vel), s)
        assert hc.tolist() == [1, 0]
        np.testing.assert_allclose(hs, [-2.0 * u, 0.0], rtol=1e-12)
    for first in (0.01, 3.0e-154, 2.9e-154):  # either side of the line above which tiny distances are not looked for
        want = [int(d > first), 0]
        assert clm.pairwise(clm.RadialHistogram(np.array([first, 0.5, 1.0]), *vel), s)[0].tolist() == want
    s.close()
