"""The sort at the edges of its tiles (1,536 keys below 450,000 bodies, 6,144
from there on) and of the rule between them: the sorted codes and the
permutation are numpy's stable sort of the same codes, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n", [1, 2, 511, 512, 1535, 1536, 1537, 3073, 49152, 449999, 450000, 450001])
def test_stable_sort_of_the_codes(bh, orc, n, bits):
    sim = bh.Simulation(bh.Config(mortonBits=bits, mortonDomain="bbox"))
    sim.setNumBodies(n)
    sim.setScenario("gaussian-mixture", 3)  # 1% duplicates: equal keys keep their order
    _, pos, _ = sim.download()
    sim.computeAccelerations()
    codes = sim.read_buffer("morton_codes", np.uint64 if bits == 64 else np.uint32, n)
    ids = sim.read_buffer("body_indices", np.uint32, n)
    want, _ = orc.morton(orc.params_from_config(sim.config), pos)
    sim.close()
    order = np.argsort(want, kind="stable")
    assert np.array_equal(ids, order.astype(np.uint32))
    assert np.array_equal(codes.astype(np.uint64), want[order].astype(np.uint64))


@pytest.mark.parametrize("systems", [1, 2, 256, 257])
def test_stable_sort_of_an_ensemble(bh, orc, systems):
    """4, 5 and 6 passes (one per byte in use: 32 code bits and the system id);
    an odd number starts in the other buffer.  Sorted codes, permutation and
    codes of every system are numpy's, bit for bit."""
    sizes = [256 + (37 * k) % 301 for k in range(systems)]
    cfg = bh.Config(walk="group", softening="plummer", plummerEps=1e-3, mortonDomain="bbox")
    ens = bh.Ensemble(sizes, cfg)
    ens.setScenarios(None, seed=2)
    _, pos, _ = ens.download()
    ens.computeAccelerations()
    n, off = int(sum(sizes)), ens.offsets
    codes = ens.read_buffer("morton_codes", np.uint64, n)
    ids = ens.read_buffer("body_indices", np.uint32, n)
    ens.close()
    p = orc.params_from_config(cfg)
    want = np.concatenate([(np.uint64(k) << np.uint64(32))
                           | orc.morton(p, pos[off[k]:off[k + 1]])[0].astype(np.uint64)
                           for k in range(systems)])
    order = np.argsort(want, kind="stable")
    assert np.array_equal(ids, order.astype(np.uint32))
    assert np.array_equal(codes, want[order])
