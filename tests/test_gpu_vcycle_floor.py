"""The mixed method on the boxes that multigrid solves, with a target beyond what
FP64 can hold: the solve runs to its iteration limit and stays on its floor.

The floor is the rounding of b - K p: at most 8 eps |K| |p| with |K| <= 12 (unit
spacing), in the 2-norm of the box.
"""
import numpy as np
import pytest

import rheon_b200 as R

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MAXF = 1.7976931348623157e308
EPS = 2.220446049250313e-16


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available() or R.device_count() == 0:
        pytest.skip("no B200")
    yield


@pytest.mark.parametrize("seeded", [False, True], ids=["cold", "seeded"])
@pytest.mark.parametrize("n,limit", [((8, 8, 8), 30), ((8, 8, 8), 120), ((5, 7, 3), 40), ((2, 2, 2), 40),
                                     ((600, 20, 20), 100), ((600, 20, 20), 250), ((520, 8, 8), 400)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_a_solve_past_its_floor_stays_there(n, limit, seeded):
    g = R.GridGeometry(n)
    b = np.random.default_rng(1).standard_normal(g.cell_len())
    b -= b.mean()
    b -= b.sum() / b.size
    ws = R.PressureWorkspace(g, 1 << 40, R.PressureImplementation.MG_MIXED)
    kw = {}
    if seeded:
        kw["initial"] = np.random.default_rng(2).standard_normal(b.size)
        kw["initial"][0] = 0.0
    with pytest.raises(R.PressureError) as e:
        ws.solve_rhs(R.PressureOperator(g, 1.0), b, 0.25, R.PressureSettings(1e-30, 0.0, MAXF, limit), **kw)
    assert e.value.kind == "IterationLimit" and e.value.iterations == limit
    assert e.value.report.true_residual_l2 <= 8 * EPS * 12 * np.linalg.norm(ws.pressure())


def test_a_batched_box_of_the_v_cycle_with_a_fixed_number_of_iterations():
    n = (64, 48, 32)

    def stepped(rel, limit, params):
        cfg = R.CarrierConfig.mixed(pressure=R.PressureSettings(rel, 0.0, MAXF, limit))
        batch = R.BatchedCarriers([R.GridGeometry(n)], cfg)
        from rheon_b200 import workloads as W

        batch.upload(0, W.fourier_faces(n, seed=3, dtype=np.float32))
        (status, rep), = batch.step(params)
        assert status == 0
        p, f = batch.pressure(0), batch.download(0)
        batch.close()
        return rep, p, f

    _, want, _ = stepped(1e-10, 1000, R.StepParams(MAXF, cfl=0.5))
    rep, p, _ = stepped(1e-30, 150, R.StepParams(MAXF, cfl=0.5, iteration_limit_ok=True))
    assert rep.pressure.iterations == 150
    # both are the solution to their residual: 1e-10 of it, times the condition
    # of the box (2 10^3)
    assert np.linalg.norm(p - want) <= 1e-6 * np.linalg.norm(want)
