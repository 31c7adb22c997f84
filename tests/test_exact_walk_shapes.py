"""The reference-semantics walk at the edges of its launch shapes: 4 bodies a
warp below 24,576 bodies, 16 from there on (partly filled last warps, one
body, leaf buckets, both softenings), against the oracle's per-body walk.

Tolerance: both sides sum the same FP32 terms (a body's accepted nodes are
decided by the same FP32 test), each term off by a few roundings and one
approximate reciprocal square root cubed (< 1e-6 relative), so a body's
difference is at most 1e-5 of the sum of its terms' magnitudes; bodies whose
theta test lies within rounding of the limit may take another node: at most
1% of the bodies, as in the parity tests.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(bh, orc, n, scenario, **cfg):
    sim = bh.Simulation(bh.Config(**cfg))
    sim.setNumBodies(n)
    sim.setScenario(scenario, 17)
    mass, pos, vel = sim.download()
    acc = sim.computeAccelerations().astype(np.float64)
    ref = orc.State(orc.params_from_config(sim.config), mass, pos, vel).accelerations()
    sim.close()
    ref = ref.astype(np.float64)
    err = np.linalg.norm(acc - ref, axis=1)
    size = np.maximum(np.linalg.norm(ref, axis=1), np.median(np.linalg.norm(ref, axis=1)))
    assert np.isfinite(acc).all()
    assert (err > 1e-5 * size).mean() <= 0.01, (err / size).max()


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 15, 17, 129, 24575, 24576, 24577, 24591])
def test_edges_of_the_body_ranges(bh, orc, n):
    if n == 1:
        sim = bh.Simulation(bh.Config())
        sim.setNumBodies(1)
        assert (sim.computeAccelerations() == 0).all()
        sim.close()
        return
    _check(bh, orc, n, "default")


@pytest.mark.parametrize("n", [5, 1003, 25001])
@pytest.mark.parametrize("cfg", [
    dict(leafSize=8, softening="plummer", mortonDomain="bbox", bhTheta=0.5),
    dict(leafSize=64, bhTheta=0.7),
    dict(mortonBits=64, softening="plummer", plummerEps=1e-4, bhTheta=0.3),
], ids=["buckets8-plummer", "buckets64-reference", "64bit"])
def test_buckets_and_softenings(bh, orc, n, cfg):
    _check(bh, orc, n, "two-clusters", **cfg)
