"""Few groups: a block's warps share one group's lists (fewer than 8 groups per
SM, and two warps below 16 where the caller waits for the forces; a group
holds about 0.7 of its 32 x bodiesPerLane bodies).  Body counts on
both sides of the rule and every block shape against the oracle's walk of the
same groups: the interactions are the same, FP32 terms within 1e-6, so sums
within 1e-5 of the larger of the body's and the median acceleration for all
but 1% of the bodies (cancelling sums).  The warps' shares are added in a fixed
order, so a repeated evaluation gives the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CFG = dict(walk="group", mortonDomain="bbox", softening="plummer", plummerEps=1e-3, bhTheta=0.7,
           leafSize=8)


def _edge(bpl, per_sm):
    import torch
    return int(0.7 * 32 * bpl * per_sm * torch.cuda.get_device_properties(0).multi_processor_count)


@pytest.mark.parametrize("bpl,per_sm", [(1, 8), (2, 8), (1, 16)])
@pytest.mark.parametrize("off", [-1, 1])
@pytest.mark.parametrize("far", [0.0, 0.4])
def test_walk_on_both_sides_of_the_rule(bh, orc, bpl, per_sm, off, far):
    sim = bh.Simulation(bh.Config(**CFG, bodiesPerLane=bpl, farAlpha=far))
    sim.setNumBodies(_edge(bpl, per_sm) + off)
    sim.setScenario("uniform-disk-kepler", 3)
    mass, pos, vel = sim.download()
    acc = sim.computeAccelerations().astype(np.float64)
    assert np.array_equal(acc, sim.computeAccelerations().astype(np.float64))  # same sums every time
    ref = orc.State(orc.params_from_config(sim.config), mass, pos, vel).accelerations()
    sim.close()
    ref = ref.astype(np.float64)
    size = np.linalg.norm(ref, axis=1)
    err = np.linalg.norm(acc - ref, axis=1) / np.maximum(size, np.median(size))
    assert (err > 1e-5).mean() <= 0.01, err.max()


@pytest.mark.parametrize("walk_block", [64, 128, 256])
@pytest.mark.parametrize("n", [2, 40, 300, 5000])
def test_every_block_shape_shares_groups(bh, orc, n, walk_block):
    sim = bh.Simulation(bh.Config(**CFG, bodiesPerLane=2, walkBlock=walk_block, farAlpha=0.4))
    sim.setNumBodies(n)
    sim.setScenario("colliding-disks", 4)
    mass, pos, vel = sim.download()
    acc = sim.computeAccelerations().astype(np.float64)
    ref = orc.State(orc.params_from_config(sim.config), mass, pos, vel).accelerations()
    sim.close()
    ref = ref.astype(np.float64)
    size = np.linalg.norm(ref, axis=1)
    err = np.linalg.norm(acc - ref, axis=1) / np.maximum(size, np.median(size))
    assert (err > 1e-5).mean() <= 0.01, err.max()
