"""The mixed method's direct solve in units far from 1. Its transforms scale the
residual by a power of two, so a right-hand side times 2^k has the pressure times
2^k, bit for bit, with the same iterations, as long as FP32 holds the residuals
and corrections themselves as normal numbers (about 1e-30 to 1e35 here). Near the
ends of FP32 a solve still reaches its target, as with the V-cycle: 1e-36 and 1e34
(1e33 for the longest box's smooth right-hand side, whose pressure is 1e4 times
larger).
"""
import numpy as np
import pytest

import rheon_b200 as R

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MAXF = 1.7976931348623157e308
SIZES = [(64, 64, 64), (33, 20, 18), (200, 40, 24)]


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


def setup(n):
    g = R.GridGeometry(n)
    return (R.PressureWorkspace(g, 1 << 40, R.PressureImplementation.MG_MIXED), R.PressureOperator(g, 1.0),
            R.PressureSettings(1e-8, 0.0, MAXF, 50))


@pytest.mark.parametrize("seeded", [False, True], ids=["cold", "seeded"])
@pytest.mark.parametrize("smooth", [False, True], ids=["noise", "smooth"])
@pytest.mark.parametrize("n", SIZES, ids=lambda n: "x".join(map(str, n)))
def test_a_scaled_right_hand_side_has_the_scaled_pressure(n, smooth, seeded):
    ws, op, st = setup(n)
    b = rhs(n, smooth)
    p0 = np.random.default_rng(2).standard_normal(b.size)
    p0[0] = 0.0

    def solve(k):
        kw = {"initial": np.ldexp(p0, k)} if seeded else {}
        return ws.solve_rhs(op, np.ldexp(b, k), 0.25, st, **kw).iterations, ws.pressure()

    its, p = solve(0)
    for k in (-80, -7, 3, 70, 100):
        its_k, p_k = solve(k)
        assert its_k == its, k
        assert np.array_equal(p_k, np.ldexp(p, k)), k


@pytest.mark.parametrize("smooth", [False, True], ids=["noise", "smooth"])
@pytest.mark.parametrize("n", SIZES, ids=lambda n: "x".join(map(str, n)))
def test_right_hand_sides_near_the_ends_of_fp32_are_solved(n, smooth):
    ws, op, st = setup(n)
    b = rhs(n, smooth)
    norm = np.linalg.norm(b)
    top = 1e33 if smooth and max(n) > 64 else 1e34
    for unit in (1e-36, 1e-34, top):
        rep = ws.solve_rhs(op, unit * b, 0.25, st)
        # the acceptance itself: the true FP64 residual
        assert rep.true_residual_l2 <= 1e-8 * norm * unit * (1 + 1e-12)
        assert rep.iterations <= 6


@pytest.mark.parametrize("n", SIZES, ids=lambda n: "x".join(map(str, n)))
def test_right_hand_sides_that_fp32_cannot_hold_break_down(n):
    # as with the V-cycle: not a run to the iteration limit
    ws, op, st = setup(n)
    for unit in (1e-100, 1e-46, 1e-42, 1e-39, 1e100):
        with pytest.raises(R.PressureError) as e:
            ws.solve_rhs(op, unit * rhs(n, False), 0.25, st)
        assert e.value.kind == "Breakdown", unit
