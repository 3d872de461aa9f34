"""A set with an over-full cell among other sets and steps: the other set of the handle keeps its small build, the set
itself returns to it when its cells are emptier again, and every step's pairs equal the oracle's.  The builds are told
apart by the launches of a step (two for few particles, three through buckets)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOX = dict(unitcell=[20.0] * 3, cutoff=1.0)


def launches(s):
    n = C.c_int64()
    assert s._handle.L.clm_stats(s._handle.h, C.byref(n)) == 0
    return n.value


def crowded(rng, n, blob):
    x = 20.0 * rng.random((n, 3))
    x = x[np.abs(x - 10.5).max(1) > 0.6]
    return np.concatenate([x, 10.3 + 0.2 * rng.random((blob, 3))])


def step(clm, orc, s, **p):
    """Launches of one step whose capacities are known, after its pairs have been checked."""
    ref = orc.run("count", p["xpositions"], p.get("ypositions"), **BOX)["count"]
    s.update(**p)
    assert clm.pairwise(clm.Count(), s) == ref
    s.update(**p)
    before = launches(s)
    assert clm.pairwise(clm.Count(), s) == ref
    return launches(s) - before


@pytest.mark.parametrize("blob", [129, 250])
def test_one_set(clm, orc, blob):
    rng = np.random.default_rng(blob)
    flat = 20.0 * rng.random((20000, 3))
    s = clm.ParticleSystem(xpositions=flat, **BOX)
    small = step(clm, orc, s, xpositions=flat)
    assert step(clm, orc, s, xpositions=crowded(rng, 20000, blob)) > small
    assert step(clm, orc, s, xpositions=flat + 0.3) == small
    assert step(clm, orc, s, xpositions=crowded(rng, 20000, 100)) == small
    s.close()


@pytest.mark.parametrize("which", ["xpositions", "ypositions"])
def test_the_other_set_keeps_its_build(clm, orc, which):
    rng = np.random.default_rng(4)
    p = {"xpositions": 20.0 * rng.random((15000, 3)), "ypositions": 20.0 * rng.random((9000, 3))}
    s = clm.ParticleSystem(**p, **BOX)
    step(clm, orc, s, **p)
    other = "ypositions" if which == "xpositions" else "xpositions"
    s.update(**{other: p[other]})
    alone = launches(s)
    clm.pairwise(clm.Count(), s)
    alone = launches(s) - alone
    p[which] = crowded(rng, 15000, 200)
    step(clm, orc, s, **p)
    s.update(**{other: p[other]})  # the set whose cells fit, by itself
    before = launches(s)
    clm.pairwise(clm.Count(), s)
    assert launches(s) - before == alone
    s.close()
