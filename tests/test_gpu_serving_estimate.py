"""The bytes that the serving pool makes room for before it creates a mixed
carrier: no fewer than the carrier takes, and no more than a tenth (and the
estimate's 1 MiB for scalars and partials) above them.
"""
import pytest

import rheon_b200 as R
from rheon_b200 import serving as S

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available() or R.device_count() == 0:
        pytest.skip("no B200")
    yield


@pytest.mark.parametrize("more", [{}, {"with_tracer": True}, {"warm_start": True}], ids=["plain", "tracer", "warm"])
@pytest.mark.parametrize("edge", [16, 64, 200])
def test_the_estimate_of_a_mixed_carrier_is_close_above_its_bytes(edge, more):
    cfg = R.CarrierConfig.mixed(**more)
    sim = R.CarrierSimulation(R.GridGeometry((edge,) * 3), cfg)
    actual, estimate = sim.allocated_bytes(), S.carrier_bytes_estimate(edge, cfg)
    sim.close()
    assert actual <= estimate <= 1.1 * actual + (1 << 20)
