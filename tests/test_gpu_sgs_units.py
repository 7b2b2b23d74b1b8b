"""The lexicographic SGS sweeps at the edges of their units of lines along x
(16 along y, 8 along z) and of their 16-step chunks: lines shorter than a
chunk, one-cell axes, units with one line, many units.

The sweeps do the serial sweep's operations in the serial order, so a solve
takes the oracle's iterations; only the sums of r.z and d.q are rounded
differently (within some ulps), which the solve's 1e-12 allows for.
"""
import numpy as np
import pytest

import oracle as O
import rheon_b200 as R

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MAXF = 1.7976931348623157e308
SIZES = [(2, 1, 1), (1, 17, 1), (1, 1, 9), (1, 40, 40), (5, 16, 8), (2, 33, 16), (15, 15, 7), (16, 31, 25), (17, 3, 40),
         (40, 48, 8), (33, 18, 10), (300, 2, 2), (129, 17, 17)]


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available() or R.device_count() == 0:
        pytest.skip("no B200")
    yield


@pytest.mark.parametrize("n", SIZES, ids=lambda n: "x".join(map(str, n)))
def test_sgs_solve_is_the_oracles_at_unit_edges(n):
    h = (0.1, 0.12, 0.15)
    g = R.GridGeometry(n, h)
    b = np.random.default_rng(sum(n)).standard_normal(g.cell_len())
    b -= b.mean()
    b -= b.sum() / b.size
    ref = O.solve_rhs(O.grid(n, h), 1.0, O.SGS_PCG_V1, b, 0.25, O.settings(1e-10, 0.0, MAXF, 5000))
    assert ref.status == O.OK
    ws = R.PressureWorkspace(g, 1 << 34, R.PressureImplementation.SGS_PCG_V1)
    # the second solve finds the first one's words and directions in the buffers
    for _ in range(2):
        rep = ws.solve_rhs(R.PressureOperator(g, 1.0), b, 0.25, R.PressureSettings(1e-10, 0.0, MAXF, 5000))
        assert rep.iterations == ref.report.iterations
        p = ws.pressure()
        assert np.linalg.norm(p - ref.pressure) <= 1e-12 * np.linalg.norm(ref.pressure)
