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
