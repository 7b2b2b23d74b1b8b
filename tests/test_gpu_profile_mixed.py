"""The timing run of the mixed method, whose solver has no z and no second
direction where it solves by fast diagonalisation: boxes whose rows the TMA path
takes, boxes that it does not take, and one that multigrid solves.
"""
import numpy as np
import pytest

import rheon_b200 as R

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MAXF = 1.7976931348623157e308


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available() or R.device_count() == 0:
        pytest.skip("no B200")
    yield


@pytest.mark.parametrize("n", [(64, 64, 64), (36, 10, 10), (33, 20, 18), (520, 16, 16)],
                         ids=lambda n: "x".join(map(str, n)))
def test_the_direction_pass_is_timed_and_solves_go_on(n):
    g = R.GridGeometry(n)
    b = np.random.default_rng(1).standard_normal(g.cell_len())
    b -= b.mean()
    b -= b.sum() / b.size
    ws = R.PressureWorkspace(g, 1 << 40, R.PressureImplementation.MG_MIXED)
    op, st = R.PressureOperator(g, 1.0), R.PressureSettings(1e-8, 0.0, MAXF, 200)
    its = ws.solve_rhs(op, b, 0.25, st).iterations
    p = ws.pressure()
    for _ in range(2):
        assert ws.profile(0, 3) > 0.0
    # the timing run leaves the solver's scalars in its own state; the next solve resets them
    assert ws.solve_rhs(op, b, 0.25, st).iterations == its
    assert np.array_equal(ws.pressure(), p)
    with pytest.raises(R.PressureError):
        ws.profile(1, 3)
