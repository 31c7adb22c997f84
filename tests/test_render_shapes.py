"""The splat and the tone table at their edges: canvases whose
size is no multiple of four (the tone map's vectors), one-pixel and tiny canvases, discs clipped at every side,
small discs beside large ones, against the oracle's FP64 density (1e-5
relative, as in the render tests, plus one weight on a disc's rim, 0.1 e^-10,
where |uv| <= 1 rounds the other way) and its tone map of the same density."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(1, 1), (3, 2), (5, 7), (64, 64), (101, 33), (1001, 77),
                                          (2, 301), (257, 255)])
@pytest.mark.parametrize("scenario", ["default", "planetary-disk"])
def test_density_and_image(bh, orc, width, height, scenario):
    sim = bh.Simulation(bh.Config())
    sim.setNumBodies(3000)
    sim.setScenario(scenario, 8)
    _, pos, _ = sim.download()
    radius = sim.read_buffer("radius_multiplier", np.float32, 3000)
    with bh.Renderer(sim, width, height) as r:
        r.setCamera(0.3, -0.2, 6.0 * width / height, 6.0)
        r.frame()
        density, image = r.readDensity(), r.readImage()
        cam = r.camera
    sim.close()
    ref = orc.render_density(cam, width, height, pos, radius)
    assert np.all(np.abs(density - ref) <= 1e-5 * ref + 5e-6)
    want = orc.tone_map(density)
    off = np.abs(image.astype(int) - want.astype(int))
    assert off.max() <= 1 and (off > 0).mean() <= 1e-3 + 4.0 / off.size
