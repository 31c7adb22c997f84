"""The build on both sides of the size from which a block packs its climbing
threads (131,072 bodies), with full and ragged last blocks of 128 slots, long
chains (duplicates: bodies at the same place) and both node layouts, against
the oracle: codes, permutation, parents, children, boxes and lengths bit for
bit; masses and centres within 1e-5 (fp32 sums in another order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [
    dict(walk="group", mortonBits=64, softening="plummer", plummerEps=1e-4),
    dict(mortonDomain="bbox", softening="plummer"),
], ids=["group-64bit", "reference-layout-32bit"])
@pytest.mark.parametrize("n", [131071, 131072, 131073, 131072 + 128])
def test_tree_around_the_packing_size(bh, orc, n, cfg):
    sim = bh.Simulation(bh.Config(**cfg))
    sim.setNumBodies(n)
    sim.setScenario("gaussian-mixture", 7)
    mass, pos, vel = sim.download()
    pos[1000:1400] = pos[1000]  # 400 bodies at one place: ordered by index alone
    sim.upload(mass, pos, vel)
    sim.computeAccelerations()
    t = sim.tree()
    codes, ids = orc.sort(*orc.morton(orc.params_from_config(sim.config), pos))
    left, right, parent = orc.build(codes, sim.config.mortonBits)
    com, m, aabb, length = orc.fill(ids, mass, pos, left, right, parent)
    sim.close()
    assert np.array_equal(t["codes"].astype(np.uint64), codes)
    assert np.array_equal(t["ids"], ids)
    assert np.array_equal(t["parent"], parent)
    assert np.array_equal(t["children"][:, 0], left[: n - 1])
    assert np.array_equal(t["children"][:, 1], right[: n - 1])
    assert np.array_equal(t["aabb"], aabb[: n - 1])
    assert np.array_equal(t["node4"][:, 3], length)
    assert np.all(np.abs(t["node4"][:, 2] - m) <= 1e-5 * np.abs(m))
    assert np.all(np.abs(t["node4"][:, :2] - com).max(1) <= 1e-5 * (np.abs(com).max(1) + length))
