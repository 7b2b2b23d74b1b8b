"""The passes of a step around its solve at the edges of their paths: rows of a
multiple of 4 cells (quads marched along z) and others, one-cell axes, boxes
smaller than a warp's line, and solves that end before their first iteration.

A projection takes the uploaded faces as the provisional velocity, so its
result is, bit for bit, the chain of the public primitives: the right-hand
side, the solve and the in-place correction do the same operations on every
value, and the sums only decide when the solve stops.
"""
import numpy as np
import pytest

import rheon_b200 as R

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MAXF = 1.7976931348623157e308
MG, JACOBI = R.PressureImplementation.MG_MIXED, R.PressureImplementation.JACOBI_PCG_V1
SIZES = [(4, 1, 1), (1, 4, 3), (4, 4, 5), (8, 3, 1), (12, 9, 33), (13, 9, 33), (32, 7, 18), (36, 40, 5), (127, 3, 4),
         (128, 5, 66), (132, 2, 3), (256, 6, 40)]


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available() or R.device_count() == 0:
        pytest.skip("no B200")
    yield


def faces(n, dtype, seed, walls=True):
    rng = np.random.default_rng(seed)
    out = []
    for d in range(3):
        shape = [n[2], n[1], n[0]]
        shape[2 - d] += 1
        f = rng.uniform(-1.0, 1.0, shape)
        if walls:
            lo = [slice(None)] * 3
            lo[2 - d] = [0, -1]
            f[tuple(lo)] = 0.0
        out.append(np.ascontiguousarray(f.reshape(-1).astype(dtype)))
    return out


def cuda(arrays):
    return [torch.from_numpy(a.copy()).cuda() for a in arrays]


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("method,storage", [(MG, "f32"), (JACOBI, "f64"), (JACOBI, "f32")],
                         ids=["mixed", "plain64", "plain32"])
@pytest.mark.parametrize("n", SIZES, ids=lambda n: "x".join(map(str, n)))
def test_projection_is_the_chain_of_the_primitives(n, method, storage):
    h, dt, density = (0.5, 0.75, 1.25), 0.125, 2.0
    dtype = np.float32 if storage == "f32" else np.float64
    g = R.GridGeometry(n, h)
    settings = R.PressureSettings(1e-9, 0.0, MAXF, 20000)
    sim = R.CarrierSimulation(g, R.CarrierConfig(density=density, pressure=settings, storage=storage,
                                                 implementation=method, fp32_advection=method is MG))
    op = R.PressureOperator(g, density)
    ws = R.PressureWorkspace(g, 1 << 40, method)
    b = torch.empty(g.cell_len(), dtype=torch.float64, device="cuda")
    # the second projection finds the first one's pressure in the buffers; the
    # third is of faces that are zero, where p = 0
    for seed in (1, 2, None):
        f = faces(n, dtype, seed) if seed else [np.zeros(g.face_len(d), dtype) for d in range(3)]
        sim.upload(f)
        rep = sim.project(dt)
        dev = cuda(f)
        op.build_rhs(dev, dt, b)
        wrep = ws.solve_rhs(op, b, dt, settings)
        p = ws.pressure()
        op.correct_candidate_in_place(torch.from_numpy(p).cuda(), dt, dev)
        assert rep.pressure.iterations == wrep.iterations
        assert np.array_equal(sim.pressure(), p)
        got = sim.download()
        want = [d.cpu().numpy() for d in dev]
        assert same(got, want)
        if seed is None:
            assert not p.any() and rep.pressure.iterations == 0
        # the report's divergence and rate are of the stored faces
        div = torch.empty_like(b)
        op.divergence(dev, div)
        assert rep.actual_divergence_max == float(div.abs().max())
        rate = sum(float(np.abs(w).max(initial=0.0)) / s for w, s in zip(want, h))
        assert rep.velocity_rate == pytest.approx(rate, rel=4e-16 * 4, abs=0.0)


@pytest.mark.parametrize("n", [(1, 1, 9), (5, 1, 7), (16, 9, 3), (31, 33, 17), (48, 20, 24)],
                         ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("h", [(1.0, 1.0, 1.0), (0.25, 1.5, 0.7)])
def test_fp32_advection_of_a_mixed_step(n, h):
    """One step of the mixed carrier against the same step in FP64. A sample in
    FP32 is off by its position's rounding, (n + 16) half ulps of a cell where
    a velocity falls by at most 2 max|u| a cell along each of 3 axes, and the
    projection does not enlarge the l2 norm of that; the two solves leave at
    most their target 1e-9 |div u| times the box's length in cells."""
    f = faces(n, np.float32, 7)
    tracer = np.random.default_rng(8).uniform(0.0, 1.0, n[0] * n[1] * n[2]).astype(np.float32)
    g = R.GridGeometry(n, h)
    settings = R.PressureSettings(1e-9, 0.0, MAXF, 200)
    out = []
    for fp32 in (False, True):
        sim = R.CarrierSimulation(g, R.CarrierConfig(pressure=settings, storage="f32", implementation=MG, max_courant=2.0,
                                                     with_tracer=True, fp32_advection=fp32))
        sim.upload(f, tracer)
        rep = sim.step(R.StepParams(MAXF, cfl=0.9))
        fs, tr = sim.download(with_tracer=True)
        out.append((np.concatenate(fs).astype(np.float64), tr.astype(np.float64)))
    size = max(n)
    position = 6 * (size + 16) * 2.0 ** -24
    (a, ta), (b, tb) = out
    top = max(np.abs(x).max(initial=0.0) for x in f)
    solve = 2 * 1e-9 * 2 * 3 ** 0.5 * np.linalg.norm(np.concatenate(f)) * size * (max(h) / min(h)) ** 2
    bound = (position + 2.0 ** -23) * top * a.size ** 0.5 + solve
    assert np.linalg.norm(a - b) <= bound
    # the tracer moves in the stepped velocity: its own positions also carry
    # that velocity's difference
    moved = rep.dt / min(h) * np.abs(a - b).max(initial=0.0)
    assert np.linalg.norm(ta - tb) <= (position + 2.0 ** -23 + 3 * moved) * ta.size ** 0.5


@pytest.mark.parametrize("bad", ["nan", "inf", "wall"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [(1, 1, 1), (7, 5, 3), (40, 33, 30)], ids=lambda n: "x".join(map(str, n)))
def test_primitives_leave_their_outputs_on_a_refused_input(n, dtype, bad):
    """The validation runs inside the operation's own launches: a refused field
    changes no output of the ones that promise it, whichever value is bad."""
    g = R.GridGeometry(n, (1.0, 1.0, 1.0))
    op = R.PressureOperator(g, 1.0)
    for axis in range(3):
        f = faces(n, dtype, 3)
        # the last face of the axis, a wall face
        f[axis][-1] = {"nan": np.nan, "inf": -np.inf, "wall": 0.5}[bad]
        dev = cuda(f)
        out = [torch.full_like(x, 7.0) for x in dev]
        kind = "NonZeroWallVelocity" if bad == "wall" else "NonFiniteInput"
        if bad != "wall":  # advection takes any wall value
            with pytest.raises(R.OperatorError, match=kind):
                R.advect_velocity(g, dev, 0.1, out)
            assert all(bool((x == 7.0).all()) for x in out)
        with pytest.raises(R.OperatorError, match=kind):
            op.build_rhs(dev, 0.1, torch.empty(g.cell_len(), dtype=torch.float64, device="cuda"))
        keep = [x.clone() for x in dev]
        with pytest.raises(R.OperatorError, match=kind):
            op.correct_candidate_in_place(torch.zeros(g.cell_len(), dtype=torch.float64, device="cuda"), 0.1, dev)
        assert all(torch.equal(x.view(torch.uint8), y.view(torch.uint8)) for x, y in zip(dev, keep))
