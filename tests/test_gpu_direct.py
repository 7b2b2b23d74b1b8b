"""The mixed method's direct preconditioner (fast diagonalisation) at the edges
of its transform tiles: axis lengths around the multiples of 4, 8 and 32 lines
and outputs, odd lengths, one-cell axes, the longest axis, uneven spacings, and
the sizes just outside it, which stay with multigrid.

Each solve's residual b - K p is recomputed here in FP64 by differences of the
pressure, so the tolerance is the solve's own target plus the rounding of that
recomputation: 8 eps (|K| |p|) per cell, |K| <= 12 times the largest weight.
"""
import numpy as np
import pytest

import rheon_b200 as R

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MAXF = 1.7976931348623157e308
MG = R.PressureImplementation.MG_MIXED


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available() or R.device_count() == 0:
        pytest.skip("no B200")
    yield


def apply_k(p, h):
    """K p of the sealed box (density 1), arrays [k][j][i]."""
    q = np.zeros_like(p)
    area = (h[1] * h[2], h[0] * h[2], h[0] * h[1])
    for d in range(3):
        diff = np.diff(p, axis=2 - d) * (area[d] / h[d])
        lo = [(0, 0)] * 3
        hi = [(0, 0)] * 3
        lo[2 - d], hi[2 - d] = (0, 1), (1, 0)
        q += np.pad(diff, hi) - np.pad(diff, lo)
    return q


def case(n, seed):
    rng = np.random.default_rng(seed)
    b = rng.standard_normal((n[2], n[1], n[0]))
    return b - b.mean()


def check(n, h, rel, seed, initial=False):
    b = case(n, seed)
    b -= b.sum() / b.size
    g = R.GridGeometry(n, h)
    ws = R.PressureWorkspace(g, 1 << 40, MG)
    kw = {}
    if initial:
        p0 = np.random.default_rng(seed + 1).standard_normal(b.size)
        p0[0] = 0.0
        kw["initial"] = p0
    rep = ws.solve_rhs(R.PressureOperator(g, 1.0), b.reshape(-1), 0.25, R.PressureSettings(rel, 0.0, MAXF, 200), **kw)
    p = ws.pressure()
    assert p[0] == 0.0
    p = p.reshape(b.shape)
    area = (h[1] * h[2], h[0] * h[2], h[0] * h[1])
    round_off = 8 * 2.3e-16 * 12 * max(a / s for a, s in zip(area, h)) * np.linalg.norm(p)
    left = np.linalg.norm(b - apply_k(p, h))
    assert left <= rel * np.linalg.norm(b) + round_off
    assert abs(left - rep.true_residual_l2) <= round_off
    return rep.iterations


EDGES = [(8, 9, 1), (16, 15, 17), (31, 33, 32), (24, 47, 49), (63, 48, 65), (96, 36, 7), (64, 97, 10), (127, 20, 128),
         (12, 129, 160), (40, 6, 255), (257, 12, 9), (6, 320, 5), (512, 4, 11), (9, 7, 511), (1, 1, 300), (13, 1, 70),
         (128, 64, 3), (3, 5, 256)]


@pytest.mark.parametrize("n", EDGES, ids=lambda n: "x".join(map(str, n)))
def test_direct_solve_meets_its_target_at_tile_edges(n):
    # two iterations reach 1e-8 on smooth data; white noise on a long axis is
    # the same within one more, and 1e-11 within two more
    assert check(n, (1.0, 1.0, 1.0), 1e-8, 3) <= 3
    assert check(n, (1.0, 1.0, 1.0), 1e-11, 4) <= 4


@pytest.mark.parametrize("h", [(0.8, 1.0, 1.25), (0.01, 0.02, 0.03), (3.0, 50.0, 7.0)])
def test_direct_solve_on_uneven_spacings(h):
    assert check((45, 32, 27), h, 1e-9, 5) <= 4


@pytest.mark.parametrize("n", [(32, 24, 40), (33, 21, 14)])
def test_seeded_direct_solve(n):
    assert check(n, (1.0, 1.0, 1.0), 1e-9, 6, initial=True) <= 4


@pytest.mark.parametrize("n,h", [((520, 8, 12), (1.0, 1.0, 1.0)), ((5, 530, 9), (1.0, 1.0, 1.0)),
                                 ((8, 8, 8), (1.0, 1.0, 1.0)), ((96, 16, 16), (1.0, 0.02, 0.02))])
def test_boxes_at_and_outside_the_direct_solves_limits_converge(n, h):
    # longer than 512 cells, no hierarchy, a condition of 2e7
    check(n, h, 1e-8, 7)


@pytest.mark.parametrize("n", [(90, 130, 130), (128, 120, 128), (56, 170, 168)], ids=lambda n: "x".join(map(str, n)))
def test_direct_solve_where_a_thread_takes_more_outputs(n):
    # more than six warps an SM: 6 or 8 outputs a thread on the axes of 90, 128
    # and 56 cells, 4 outputs on boxes of fewer lines (the edges above)
    assert check(n, (1.0, 1.0, 1.0), 1e-8, 7) <= 3
