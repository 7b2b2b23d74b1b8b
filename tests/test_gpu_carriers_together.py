"""Plain carriers stepped together: their cooperative solves share the SMs.

Boxes of one, two, three and four lanes of SMs, alone and mixed. A carrier's
step is its own whatever steps beside it: the arrays are the same bits as those
of a carrier that steps alone. Small ones overlap.
"""
import time

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


def carriers(sizes, method=R.PressureImplementation.JACOBI_PCG_V1):
    out = []
    for i, n in enumerate(sizes):
        cfg = R.CarrierConfig(pressure=R.PressureSettings(1e-8, 0.0, MAXF, 100000), storage="f64",
                              implementation=method)
        sim = R.CarrierSimulation(R.GridGeometry(n), cfg)
        sim.init_fourier(i + 1)
        out.append(sim)
    return out


@pytest.mark.parametrize("sizes", [[(16, 16, 16)] * 6, [(32, 32, 32)] * 5,
                                   [(16, 16, 16), (64, 64, 64), (17, 9, 5), (32, 32, 32), (96, 40, 48), (23, 23, 23)],
                                   [(33, 20, 48), (37, 37, 37), (63, 63, 63)], [(75, 75, 75), (128, 128, 100)]],
                         ids=["16cube", "32cube", "mixed", "longer runs", "longest runs"])
def test_a_carrier_steps_the_same_beside_others(sizes):
    # Boxes of more than two lanes take longer runs of cells a thread beside
    # others, so their sums fold in another order. The sums are compensated
    # (relative error below 1e-29), and agree to the last bit of a double.
    prm = [R.StepParams(MAXF, cfl=0.5)] * len(sizes)
    alone, together = carriers(sizes), carriers(sizes)
    for _ in range(2):
        want = [sim.step(p) for sim, p in zip(alone, prm)]
        got = R.step_all(together, prm)
        for w, (status, g) in zip(want, got):
            assert status == 0
            assert g.pressure.iterations == w.pressure.iterations
    for a, b in zip(alone, together):
        for x, y in zip(a.download(), b.download()):
            assert np.array_equal(x, y)
    for sim in alone + together:
        sim.close()


@pytest.mark.parametrize("n", [(16, 16, 16), (32, 32, 32), (33, 20, 48), (45, 45, 45)],
                         ids=["16cube", "32cube", "33x20x48", "45cube"])
def test_small_carriers_overlap(n):
    # one lane or two: four or two steps at a time, so eight take well under the
    # time of eight in a row
    sims = carriers([n] * 8)
    prm = [R.StepParams(MAXF, cfl=0.5)] * len(sims)
    ratios = []
    for _ in range(5):
        t0 = time.perf_counter()
        for sim, p in zip(sims, prm):
            sim.step(p)
        t1 = time.perf_counter()
        R.step_all(sims, prm)
        ratios.append((time.perf_counter() - t1) / (t1 - t0))
    assert min(ratios) < 0.75, ratios
    for sim in sims:
        sim.close()
