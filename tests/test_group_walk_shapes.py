"""The group walk where its packing can go wrong: one group of every fill
around the 32-body sub-slots (odd sub-slots take two list entries per packed
instruction), several groups, all group sizes, both softenings (with the
self test), without softening, monopoles, and far-field batches of fewer and
more than 64 nodes -- against the oracle's walk of the same groups.

Tolerance: the acceptance tests round identically on both sides, so every
body has the same interactions; each FP32 term is within 1e-6 of the oracle's
(a few roundings, one approximate reciprocal square root to the 7th power at
most), sums of them within 1e-5 of the larger of the body's and the median
acceleration.  At most 1% of the bodies may exceed it (cancelling sums).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BASE = dict(walk="group", mortonDomain="bbox", softening="plummer", plummerEps=1e-3, bhTheta=0.5)


def _check(bh, orc, n, scenario, limit=1e-5, **cfg):
    sim = bh.Simulation(bh.Config(**{**BASE, **cfg}))
    sim.setNumBodies(n)
    sim.setScenario(scenario, 23)
    mass, pos, vel = sim.download()
    acc = sim.computeAccelerations().astype(np.float64)
    ref = orc.State(orc.params_from_config(sim.config), mass, pos, vel).accelerations()
    sim.close()
    assert np.isfinite(acc).all()
    ref = ref.astype(np.float64)
    err = np.linalg.norm(acc - ref, axis=1)
    size = np.linalg.norm(ref, axis=1)
    size = np.maximum(size, np.median(size))
    assert (err > limit * size).mean() <= 0.01, (err / size).max()


@pytest.mark.parametrize("bpl", [1, 2, 4])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 700])
def test_fills_of_the_sub_slots(bh, orc, n, bpl):
    _check(bh, orc, n, "uniform-disk-kepler", bodiesPerLane=bpl, leafSize=4)


@pytest.mark.parametrize("bpl", [1, 2, 4])
@pytest.mark.parametrize("cfg", [
    dict(softening="reference", leafSize=8),
    dict(plummerEps=0.0, leafSize=1),
    dict(multipole=1, leafSize=2),
    dict(multipole=1, softening="reference", leafSize=4, mortonBits=64),
], ids=["reference", "unsoftened", "monopole", "monopole-reference-64bit"])
def test_softenings_and_orders(bh, orc, cfg, bpl):
    _check(bh, orc, 3001, "colliding-disks", bodiesPerLane=bpl, **cfg)


@pytest.mark.parametrize("bpl", [1, 2, 4])
@pytest.mark.parametrize("n,alpha", [(300, 0.5), (2500, 0.25), (30011, 0.4)])
def test_far_batches(bh, orc, n, alpha, bpl):
    _check(bh, orc, n, "colliding-disks", bodiesPerLane=bpl, leafSize=4, farAlpha=alpha)


@pytest.mark.parametrize("bpl", [1, 4])
@pytest.mark.parametrize("kind", ["chain", "pairs", "pile"])
@pytest.mark.parametrize("n", [3, 33, 300])
def test_tops_of_uneven_trees(bh, orc, n, kind, bpl):
    """The top five levels are walked in one step: trees with leaves and long
    chains among them (bodies at 2^-k, tight pairs of those, one cell holding
    all but one)."""
    k = np.arange(n)
    if kind == "chain":
        x = 2.0 ** -(k % 15)
        pos = np.stack([x, x * (1 + k // 15)], 1)
    elif kind == "pairs":
        x = 2.0 ** -((k // 2) % 12)
        pos = np.stack([x + 1e-4 * (k % 2), x * (1 + k // 24)], 1)
    else:
        pos = np.stack([1e-3 * (k % 17), 1e-3 * (k // 17)], 1)
        pos[0] = (1.0, 1.0)
    sim = bh.Simulation(bh.Config(**BASE, bodiesPerLane=bpl, leafSize=2))
    sim.setNumBodies(n)
    pos = pos.astype(np.float32)
    mass, vel = np.full(n, 1.0 / n, np.float32), np.zeros((n, 2), np.float32)
    sim.upload(mass, pos, vel)
    acc = sim.computeAccelerations().astype(np.float64)
    state = orc.State(orc.params_from_config(sim.config), mass, pos, vel)
    ref = state.accelerations().astype(np.float64)
    sim.close()
    size = np.linalg.norm(ref, axis=1)
    size = np.maximum(size, np.median(size))
    assert (np.linalg.norm(acc - ref, axis=1) > 1e-5 * size).mean() <= 0.01
