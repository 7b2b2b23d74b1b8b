"""The timing run of a solver keeps no device memory: what it allocates for the
call is not part of allocated_bytes().
"""
import pytest

import rheon_b200 as R

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available() or R.device_count() == 0:
        pytest.skip("no B200")
    yield


@pytest.mark.parametrize("method", [R.PressureImplementation.MG_MIXED, R.PressureImplementation.JACOBI_PCG_V1],
                         ids=["mixed", "jacobi"])
def test_a_timing_run_gives_its_memory_back(method):
    n = (160, 128, 128)  # a vector of doubles is 20 MiB
    ws = R.PressureWorkspace(R.GridGeometry(n), 1 << 40, method)
    ws.solve_rhs(R.PressureOperator(R.GridGeometry(n), 1.0), torch.zeros(n[0] * n[1] * n[2], dtype=torch.float64,
                                                                         device="cuda"), 0.25,
                 R.PressureSettings(1e-8, 0.0, 1.7976931348623157e308, 10))
    torch.cuda.synchronize()
    before, _ = torch.cuda.mem_get_info()
    assert ws.profile(0, 2) > 0.0
    after, _ = torch.cuda.mem_get_info()
    assert before - after < 8 << 20
