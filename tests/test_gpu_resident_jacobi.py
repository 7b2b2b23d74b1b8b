"""The resident Jacobi-PCG kernel against the per-pass kernels.

Both compute the same iteration cell by cell; only the order in which the
double-double partials of d.q, r.r and r.z are combined differs (about one ulp
of each scalar, 1e-16, amplified by the recurrence): per-iteration scalars and
pressures to 1e-12, as every Jacobi path against the oracle. The boxes lie at
the edges of the kernel's bricks (32 x 16 x Q cells, Q the shortest run that
gives every brick an SM): rows and lanes cut off, one-cell axes, whole and
partial runs of every length, the largest box, and one beyond it.
RB200_PERSISTENT=0 selects the per-pass kernels for a workspace made while it
is set.
"""
import os

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


def workspace(g, persistent):
    old = os.environ.get("RB200_PERSISTENT")
    try:
        if persistent:
            os.environ.pop("RB200_PERSISTENT", None)
        else:
            os.environ["RB200_PERSISTENT"] = "0"
        return R.PressureWorkspace(g, 1 << 40)
    finally:
        if old is None:
            os.environ.pop("RB200_PERSISTENT", None)
        else:
            os.environ["RB200_PERSISTENT"] = old


def rhs_of(n, scale=1.0, seed=5):
    b = np.random.default_rng(seed).standard_normal(n[0] * n[1] * n[2])
    b -= b.mean()
    b -= b.sum() / b.size
    return b * scale


def run(n, b, persistent, settings, h=(1.0, 1.0, 1.0), cap=100):
    g = R.GridGeometry(n, h)
    ws = workspace(g, persistent)
    ws.set_trace(cap)
    try:
        rep = ws.solve_rhs(R.PressureOperator(g, 1.0), b, 0.25, settings)
        return "Ok", rep.iterations, ws.trace(rep.iterations), ws.pressure()
    except R.PressureError as e:
        return e.kind, e.iterations, ws.trace(e.iterations), ws.pressure()


EDGES = [(1, 1, 7), (31, 16, 2), (33, 17, 5), (64, 15, 33), (32, 48, 1), (40, 16, 150), (5, 130, 9), (63, 48, 37),
         (96, 80, 70), (128, 96, 101), (160, 33, 128), (128, 128, 128), (161, 129, 40), (200, 128, 128)]


@pytest.mark.parametrize("n", EDGES, ids=lambda n: "x".join(map(str, n)))
def test_resident_iterations_track_the_per_pass_ones(n):
    # 80 iterations: more than one launch of the kernel
    s = R.PressureSettings(1e-13, 0.0, MAXF, 80)
    b = rhs_of(n)
    (ka, ia, ta, pa), (kb, ib, tb, pb) = run(n, b, False, s), run(n, b, True, s)
    assert (ka, ia) == (kb, ib)
    worst = 0.0
    for k in range(min(ia - 1, 60 if max(n) > 1 else 1)):
        for name in ("curvature", "alpha", "recursive_l2", "rz", "beta"):
            x, y = getattr(ta[k], name), getattr(tb[k], name)
            # a small box converges to its rounding floor, where scalars are noise
            if ta[k].recursive_l2 > 1e-9 * np.linalg.norm(b):
                worst = max(worst, abs(x - y) / abs(x))
    assert worst <= 1e-12, worst
    assert np.linalg.norm(pa - pb) <= 1e-11 * np.linalg.norm(pa)


@pytest.mark.parametrize("scale", [1e-145, 1e140])
def test_quotients_outside_the_fast_division_range(scale):
    n, s = (33, 20, 18), R.PressureSettings(0.0, 0.0, MAXF, 70)
    b = rhs_of(n, scale)
    (ka, ia, _, pa), (kb, ib, _, pb) = run(n, b, False, s), run(n, b, True, s)
    assert (ka, ia) == (kb, ib)
    assert np.max(np.abs(pa - pb)) <= 1e-10 * np.max(np.abs(pa))


def test_checks_and_restarts_as_per_pass():
    n = (64, 40, 24)
    s = R.PressureSettings(1e-14, 0.0, MAXF, 3000)
    b = rhs_of(n, seed=8)
    (ka, ia, _, pa), (kb, ib, _, pb) = run(n, b, False, s, cap=3000), run(n, b, True, s, cap=3000)
    assert (ka, ia) == (kb, ib)
    assert np.linalg.norm(pa - pb) <= 1e-11 * np.linalg.norm(pa)
