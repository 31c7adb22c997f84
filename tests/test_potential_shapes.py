"""The direct-sum potential at the edges of its tiling (256 bodies j per tile,
1,024 bodies i per block, each unordered pair once) against the oracle's FP64
sum: FP32 pair terms within 3e-7, so the sum of same-signed terms within 1e-6
relative (the bound of the diagnostics tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("softening", ["plummer", "reference"])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 1023, 1024, 1025, 1281, 2048, 4097, 9001])
def test_every_pair_once(bh, orc, n, softening):
    sim = bh.Simulation(bh.Config(softening=softening, plummerEps=1e-3))
    sim.setNumBodies(n)
    sim.setScenario("uniform-disk-kepler", 5)
    mass, pos, vel = sim.download()
    d = sim.diagnostics()
    sim.close()
    ref = orc.diagnostics_fp64(orc.params_from_config(bh.Config(softening=softening,
                                                                plummerEps=1e-3)), mass, pos, vel)
    assert d["potential_energy"] == pytest.approx(ref["potential_energy"], rel=1e-6, abs=1e-30)
    assert d["pairs"] == (n * (n - 1) // 2)


def test_coincident_and_massless_bodies_count_nothing(bh):
    # two coincident unsoftened bodies, a massless one and a distant one
    sim = bh.Simulation(bh.Config(softening="plummer", plummerEps=0.0))
    sim.setNumBodies(4)
    mass = np.array([1.0, 2.0, 0.0, 3.0], np.float32)
    pos = np.array([[0, 0], [0, 0], [1, 0], [0, 4]], np.float32)
    sim.upload(mass, pos, np.zeros((4, 2), np.float32))
    assert sim.diagnostics()["potential_energy"] == pytest.approx(-(1 + 2) * 3 / 4, rel=1e-6)
    sim.close()
