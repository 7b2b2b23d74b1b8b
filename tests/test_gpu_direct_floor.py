"""The mixed method's direct solve on uneven spacings, up to the condition of 1e9
that it covers: it reaches 1e-8 where FP64 can hold it, and past its floor it stays
there until the iteration limit.

The floor is the rounding of b - K p: at most 8 eps |K| |p| in the 2-norm (seven
products and sums a row), with |K| at most the largest eigenvalues of the three
axes together.
"""
import numpy as np
import pytest

import rheon_b200 as R

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MAXF = 1.7976931348623157e308
EPS = 2.220446049250313e-16
BOXES = [((96, 16, 16), (1.0, 0.02, 0.02)), ((64, 64, 64), (1.0, 0.0025, 1.0)), ((512, 16, 16), (1.0, 0.02, 0.02)),
         ((512, 8, 8), (1.0, 0.02, 0.02)), ((512, 3, 3), (1.0, 0.015, 0.015)), ((64, 8, 8), (1.0, 0.0019, 0.0019)),
         ((12, 4, 4), (1.0, 0.00035, 0.00035))]


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available() or R.device_count() == 0:
        pytest.skip("no B200")
    yield


def rhs(n, smooth):
    if smooth:
        x, y, z = [np.cos(np.pi * (np.arange(m) + 0.5) / m) for m in n]
        b = z[:, None, None] + y[None, :, None] + x[None, None, :]
    else:
        b = np.random.default_rng(1).standard_normal((n[2], n[1], n[0]))
    b = b - b.mean()
    b -= b.sum() / b.size
    return b.reshape(-1)


@pytest.mark.parametrize("smooth", [False, True], ids=["noise", "smooth"])
@pytest.mark.parametrize("n,h", BOXES, ids=["x".join(map(str, n)) for n, _ in BOXES])
def test_a_direct_solve_past_its_floor_stays_there(n, h, smooth):
    g = R.GridGeometry(n, h)
    b = rhs(n, smooth)
    volume = h[0] * h[1] * h[2]
    norm_k = sum(4.0 * volume / x**2 for x in h)
    ws = R.PressureWorkspace(g, 1 << 40, R.PressureImplementation.MG_MIXED)
    for limit in (40, 41, 300):
        with pytest.raises(R.PressureError) as e:
            ws.solve_rhs(R.PressureOperator(g, 1.0), b, 0.25, R.PressureSettings(1e-30, 0.0, MAXF, limit))
        assert e.value.kind == "IterationLimit" and e.value.iterations == limit
        assert e.value.report.true_residual_l2 <= 8 * EPS * norm_k * np.linalg.norm(ws.pressure())


@pytest.mark.parametrize("n,h", BOXES[:4], ids=["x".join(map(str, n)) for n, _ in BOXES[:4]])
def test_noise_is_solved_to_1e_8(n, h):
    g = R.GridGeometry(n, h)
    b = rhs(n, False)
    ws = R.PressureWorkspace(g, 1 << 40, R.PressureImplementation.MG_MIXED)
    rep = ws.solve_rhs(R.PressureOperator(g, 1.0), b, 0.25, R.PressureSettings(1e-8, 0.0, MAXF, 50))
    assert rep.true_residual_l2 <= 1e-8 * np.linalg.norm(b) * (1 + 1e-12)
