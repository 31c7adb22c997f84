"""An ensemble's groups start at their own system's root, whose index is the
system's first or last slot: every system's forces are those of a simulation
of that system alone.  The same interactions are summed in another order where
the two share groups differently: 2e-5 of the 2-norm (a thousand fp32 terms)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CFG = dict(walk="group", softening="plummer", plummerEps=1e-3, mortonDomain="bbox")


@pytest.mark.parametrize("sizes", [[256], [256, 256], [300, 5000, 256], [257 + k for k in range(300)]])
def test_each_system_is_the_simulation_of_itself(bh, sizes):
    ens = bh.Ensemble(sizes, bh.Config(**CFG))
    ens.setScenarios(None, seed=4)
    mass, pos, vel = ens.download()
    acc, off = ens.computeAccelerations(), ens.offsets
    ens.close()
    for k in sorted({0, 1, len(sizes) // 2, len(sizes) - 1} & set(range(len(sizes)))):
        sl = slice(off[k], off[k + 1])
        sim = bh.Simulation(bh.Config(**CFG))
        sim.setNumBodies(len(mass[sl]))
        sim.upload(mass[sl], pos[sl], vel[sl])
        one = sim.computeAccelerations()
        sim.close()
        assert np.linalg.norm(acc[sl] - one) <= 2e-5 * np.linalg.norm(one), k
