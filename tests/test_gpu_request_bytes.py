"""A request's admission estimate covers what its simulation comes to hold:
prepared, stepped, a frame reduced, over sizes and mixes."""
import pytest

from spatial_cell_gb300 import serving

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 4096, 30011, 262144])
@pytest.mark.parametrize("mix", [(0.4, 0.4, 0.1, 0.1), (0.01, 0.01, 0.49, 0.49), (0.97, 0.01, 0.01, 0.01)])
def test_estimate_covers_the_sim(product, n, mix):
    req = serving.Request(0, 0.0, 5, n, 2, mix)
    sim = req.start()
    sim.step(req.horizon)
    sim.sync()
    sim.reduce_frame()
    assert sim.device_bytes() <= req.bytes
    sim.close()
