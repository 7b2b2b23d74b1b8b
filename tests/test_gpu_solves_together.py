"""Cooperative solves driven from several host threads at a time: workspaces
whose kernels each take most of the SMs, and a carrier beside them. Every solve
has the bits that it has alone.
"""
import threading

import numpy as np
import pytest

import rheon_b200 as R

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MAXF = 1.7976931348623157e308
J, RB = R.PressureImplementation.JACOBI_PCG_V1, R.PressureImplementation.RBSGS_PCG
# (box, method): resident kernels of 128, 108, 64 and 16 blocks, streaming kernels
SOLVES = [((64, 64, 64), J), ((80, 48, 45), J), ((32, 32, 32), J), ((16, 16, 16), J), ((64, 64, 64), RB),
          ((160, 64, 64), J)]


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available() or R.device_count() == 0:
        pytest.skip("no B200")
    yield


def test_solves_from_several_threads_are_those_of_one():
    settings = R.PressureSettings(1e-8, 0.0, MAXF, 5000)

    def job(n, method, seed):
        g = R.GridGeometry(n)
        b = np.random.default_rng(seed).standard_normal(g.cell_len())
        b -= b.mean()
        b -= b.sum() / b.size
        return R.PressureWorkspace(g, 1 << 40, method), R.PressureOperator(g, 1.0), b

    def carrier():
        sim = R.CarrierSimulation(R.GridGeometry((48, 48, 48)), R.CarrierConfig(pressure=settings, storage="f64"))
        sim.init_fourier(3)
        return sim

    jobs = [job(n, m, i) for i, (n, m) in enumerate(SOLVES)]
    want = []
    for ws, op, b in jobs:
        rep = ws.solve_rhs(op, b, 0.25, settings)
        want.append((rep.iterations, ws.pressure()))
    alone, beside = carrier(), carrier()
    params = R.StepParams(MAXF, cfl=0.5)
    rounds = 4
    for _ in range(rounds):
        alone.step(params)
    got = [[] for _ in jobs]
    failed = []
    gate = threading.Barrier(len(jobs) + 1)

    def solve(i):
        try:
            ws, op, b = jobs[i]
            gate.wait()
            for _ in range(rounds):
                rep = ws.solve_rhs(op, b, 0.25, settings)
                got[i].append((rep.iterations, ws.pressure()))
        except Exception as e:  # noqa: BLE001
            failed.append((SOLVES[i], e))

    def step():
        try:
            gate.wait()
            for _ in range(rounds):
                beside.step(params)
        except Exception as e:  # noqa: BLE001
            failed.append(("carrier", e))

    threads = [threading.Thread(target=solve, args=(i,)) for i in range(len(jobs))] + [threading.Thread(target=step)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for (its, p), runs in zip(want, got):
        assert len(runs) == rounds
        for its2, p2 in runs:
            assert its2 == its
            assert np.array_equal(p2, p)
    for a, b in zip(alone.download(), beside.download()):
        assert np.array_equal(a, b)
