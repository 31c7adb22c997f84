"""The force VJP at the edges of its packing (two bodies per instruction, four
per reduction, 32 list entries per batch) for every group size.

theta = 0 opens every node, so the sum runs over bodies only and the FP64
direct-sum VJP is its exact value: FP32 terms within 1e-6 and sums of at most
1,100 of them (in float atomics, any order) stay within 2e-5 of the norm.
theta = 0.5 adds the node path; its truncation bounds the error (2e-2, as
for the 4,096-body case of the adjoint tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _errors(bh, orc, n, theta, bpl, leaf=8, eps=0.05):
    cfg = bh.Config(bhTheta=theta, softening="plummer", plummerEps=eps, mortonDomain="bbox",
                    integrator="leapfrog-kdk", walk="group", leafSize=leaf, bodiesPerLane=bpl)
    mass, pos, vel, _ = bh.generate_scenario("uniform-disk-kepler", n, 9)
    sim = bh.Simulation(cfg)
    sim.setNumBodies(n)
    sim.upload(mass, pos, vel)
    abar = np.random.default_rng(n).normal(size=(n, 2)).astype(np.float32)
    xb, mb = sim.force_vjp(abar)
    xr, mr = orc.force_vjp_fp64(orc.params_from_config(sim.config), mass, pos, abar)
    sim.close()
    assert np.isfinite(xb).all() and np.isfinite(mb).all()
    return (np.linalg.norm(xb - xr) / np.linalg.norm(xr),
            np.linalg.norm(mb - mr) / np.linalg.norm(mr))


@pytest.mark.parametrize("bpl", [1, 2, 4])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 31, 33, 64, 65, 127, 128, 129, 131, 1100])
def test_bodies_only_equals_the_direct_sum(bh, orc, n, bpl):
    assert max(_errors(bh, orc, n, 0.0, bpl)) <= 2e-5


@pytest.mark.parametrize("bpl", [1, 2, 4])
@pytest.mark.parametrize("leaf", [1, 8])
def test_nodes_within_their_truncation(bh, orc, bpl, leaf):
    assert max(_errors(bh, orc, 5003, 0.5, bpl, leaf, eps=1e-3)) <= 2e-2
