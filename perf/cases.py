"""The calls whose time is followed: one pass of each through the public API.

A case is a dict of plain values; its "kind" names the entry point. The boxes,
tolerances and flows are those of the benchmark and the tests: edges of 32 to
256 cells, a random-Fourier velocity (8 modes, wavenumbers 1 to 8, 0.05 noise,
wall-normal faces 0), CFL 0.5, relative residual 1e-8 (1e-12 where a pressure
itself is the result of the mixed method). Carriers, batches and liquid states
are resident: a pass advances them, as a user's time loop does, and reads the
accepted state back.
"""
import math

import torch

import rheon_b200 as R
from rheon_b200 import box_flux as B
from rheon_b200 import dense3d as D
from rheon_b200 import liquid as L

MAXF = 1.7976931348623157e308
METHODS = {"jacobi": R.PressureImplementation.JACOBI_PCG_V1, "sgs": R.PressureImplementation.SGS_PCG_V1,
           "rbsgs": R.PressureImplementation.RBSGS_PCG, "mixed": R.PressureImplementation.MG_MIXED}
# the edges of the batched boxes
EDGES = (32, 48, 64, 96, 128)


def _case(kind, n, h=(1.0, 1.0, 1.0), **more):
    return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], hx=h[0], hy=h[1], hz=h[2], **more)


def listed():
    named = {
        # the smallest call: one operator primitive on a 32^3 box, launch and call overhead
        "rhs_32": _case("rhs", (32, 32, 32), dtype="float64"),
        # semi-Lagrangian advection alone, the plain method's arithmetic
        "advect_128": _case("advect", (128, 128, 128), dtype="float64"),
        # one interval of liquid-volume transport on a ragged box
        "liquid_ragged": _case("liquid", (150, 96, 75)),
        # one exported frame of a state: the text of 96^3 cells
        "frame_96": _case("frame", (96, 96, 96)),
        # the reference's own method, a small resident box: latency of many iterations
        "step_plain_32": _case("step", (32, 32, 32), method="jacobi", storage="f64", tracer=False),
        # the headline workload: 128^3, f64, Jacobi-PCG
        "step_plain_128": _case("step", (128, 128, 128), method="jacobi", storage="f64", tracer=False),
        # the reference's second method through the pressure workspace, odd extents
        "solve_sgs_ragged": _case("solve", (63, 48, 37), method="sgs", rel=1e-8),
        # the mixed method through the pressure workspace, odd extents
        "solve_mixed_ragged": _case("solve", (90, 75, 63), method="mixed", rel=1e-12),
        # the mixed-precision carrier at the headline size
        "step_mixed_128": _case("step", (128, 128, 128), method="mixed", storage="f32", tracer=False),
        # the mixed-precision carrier at its largest size, with a buoyant tracer
        "step_mixed_256": _case("step", (256, 256, 256), method="mixed", storage="f32", tracer=True),
        # an open-boundary projection with the default method
        "box_flux_ragged": _case("box_flux", (80, 48, 45), method="jacobi"),
        # 64 uneven boxes advanced together for a few steps
        "batch_64": dict(kind="batch", boxes=64, pick=20261203, steps=4),
    }
    return [dict(c, name=k) for k, c in named.items()]


def draw(rng):
    def edge(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def box(lo, hi, cells):
        while True:
            n = (edge(lo, hi), edge(lo, hi), edge(lo, hi))
            if n[0] * n[1] * n[2] <= cells:
                return n

    h = rng.choice([(1.0, 1.0, 1.0), (1.0, 1.0, 1.0), (0.5, 0.5, 0.5), (0.8, 1.0, 1.25)])
    kind = rng.choice(["rhs", "advect", "liquid", "frame", "plain", "sgs", "mixed_solve", "mixed_step", "mixed_step",
                       "box_flux", "batch"])
    if kind == "rhs":
        return _case("rhs", box(16, 256, 4 << 20), h, dtype=rng.choice(["float64", "float32"]))
    if kind == "advect":
        return _case("advect", box(16, 200, 2 << 20), h, dtype=rng.choice(["float64", "float32"]))
    if kind == "liquid":
        return _case("liquid", box(16, 200, 2 << 20), h)
    if kind == "frame":
        return _case("frame", box(16, 128, 1 << 20))
    if kind == "plain":
        return _case("step", box(16, 96, 400000), h, method=rng.choice(["jacobi", "jacobi", "rbsgs"]), storage="f64",
                     tracer=False)
    if kind == "sgs":
        return _case("solve", box(12, 64, 100000), h, method="sgs", rel=1e-8)
    if kind == "mixed_solve":
        return _case("solve", box(16, 256, 2 << 20), h, method="mixed", rel=1e-12)
    if kind == "mixed_step":
        # carriers of the serving stream: edges that are multiples of 8
        n = box(32, 256, 6 << 20)
        return _case("step", tuple(8 * max(4, round(x / 8)) for x in n), method="mixed", storage="f32",
                     tracer=rng.random() < 0.3)
    if kind == "box_flux":
        return _case("box_flux", box(16, 80, 200000), h, method=rng.choice(["jacobi", "rbsgs", "mixed"]))
    return dict(kind="batch", boxes=rng.randint(2, 24), pick=rng.randint(1, 1 << 30), steps=rng.randint(1, 4))


# ------------------------------------------------------------------ inputs
def _size(case):
    return (case["nx"], case["ny"], case["nz"]), (case["hx"], case["hy"], case["hz"])


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _face_shape(n, a):
    s = [n[2], n[1], n[0]]
    s[2 - a] += 1
    return s


def _fourier(n, gen):
    """Three f64 face arrays [k][j][i] of a random-Fourier flow, walls 0."""
    r = torch.rand((8, 7), dtype=torch.float64, generator=gen, device="cuda").cpu()
    kv, phase = 1 + torch.floor(8 * r[:, :3]), math.pi * (2 * r[:, 3] - 1)
    amp = 2 * r[:, 4:] - 1
    amp = amp / amp.norm(dim=1, keepdim=True)
    faces = []
    for a in range(3):
        s = _face_shape(n, a)
        out = 0.1 * torch.rand(s, dtype=torch.float64, generator=gen, device="cuda") - 0.05
        for m in range(8):
            arg = float(phase[m])
            for d in range(3):
                x = torch.arange(s[2 - d], dtype=torch.float64, device="cuda") + (0.0 if d == a else 0.5)
                shape = [1, 1, 1]
                shape[2 - d] = -1
                arg = arg + (2 * math.pi * float(kv[m, d]) / n[d] * x).reshape(shape)
            out += float(amp[m, a]) * torch.sin(arg)
        out.select(2 - a, 0).zero_()
        out.select(2 - a, n[a]).zero_()
        faces.append(out)
    return faces


def _solenoidal(n, h, gen):
    """Three f32 face arrays of zero divergence up to rounding: the discrete
    curl of a smooth potential that vanishes on the walls."""
    psi = []
    for a in range(3):
        s = [n[2] + 1, n[1] + 1, n[0] + 1]
        s[2 - a] -= 1
        p = torch.ones(s, dtype=torch.float64, device="cuda")
        for d in range(3):
            x = torch.arange(s[2 - d], dtype=torch.float64, device="cuda") + (0.5 if d == a else 0.0)
            k = 1 + int(3 * float(torch.rand((), generator=gen, device="cuda")))
            shape = [1, 1, 1]
            shape[2 - d] = -1
            p = p * torch.sin(math.pi * k * x / n[d]).reshape(shape)
        psi.append(min(n) * min(h) / 8 * p)

    def diff(f, d):
        m = f.shape[2 - d] - 1
        return (f.narrow(2 - d, 1, m) - f.narrow(2 - d, 0, m)) / h[d]

    u = diff(psi[2], 1) - diff(psi[1], 2)
    v = diff(psi[0], 2) - diff(psi[2], 0)
    w = diff(psi[1], 0) - diff(psi[0], 1)
    return [f.float().contiguous() for f in (u, v, w)]


def _blob(n, gen):
    """A Gaussian density blob, f32 cells [k][j][i]."""
    c = 0.35 + 0.3 * torch.rand(3, dtype=torch.float64, generator=gen, device="cuda").cpu()
    sigma = 20.0 * min(n) / 256.0
    r2 = 0.0
    for d in range(3):
        x = torch.arange(n[d], dtype=torch.float64, device="cuda") + 0.5 - float(c[d]) * n[d]
        shape = [1, 1, 1]
        shape[2 - d] = -1
        r2 = r2 + (x * x).reshape(shape)
    return torch.exp(-r2 / (2 * sigma * sigma)).float()


def _fraction(n, gen):
    """Liquid occupancy: a ball of 0.875 in a third of the box, 0.125 around it (a
    dry surrounding would, after hundreds of passes, hold fractions that underflow)."""
    c = 0.4 + 0.2 * torch.rand(3, dtype=torch.float64, generator=gen, device="cuda").cpu()
    r2 = 0.0
    for d in range(3):
        x = torch.arange(n[d], dtype=torch.float64, device="cuda") + 0.5 - float(c[d]) * n[d]
        shape = [1, 1, 1]
        shape[2 - d] = -1
        r2 = r2 + (x * x).reshape(shape)
    return 0.125 + 0.75 * torch.clamp(min(n) / 3 + 0.5 - torch.sqrt(r2), 0.0, 1.0)


def _rhs_of(faces, h, dt):
    """Integrated divergence over dt, negated, in f64 (the pressure system's right-hand side)."""
    area = (h[1] * h[2], h[0] * h[2], h[0] * h[1])
    b = 0.0
    for a in range(3):
        m = faces[a].shape[2 - a] - 1
        b = b + area[a] * (faces[a].narrow(2 - a, 0, m).double() - faces[a].narrow(2 - a, 1, m).double())
    return b / dt


def _boxes(case):
    import random

    r = random.Random(case["pick"])
    return [(r.choice(EDGES),) * 3 for _ in range(case["boxes"])]


def _settings(rel):
    return R.PressureSettings(rel, 0.0, MAXF, 100000)


def _blank(n, dtype):
    return [torch.empty(_face_shape(n, a), dtype=dtype, device="cuda") for a in range(3)]


def _config(case):
    if case["method"] == "mixed":
        return R.CarrierConfig.mixed(pressure=_settings(1e-8), with_tracer=case["tracer"])
    return R.CarrierConfig(pressure=_settings(1e-8), storage=case["storage"], implementation=METHODS[case["method"]],
                           with_tracer=case["tracer"])


def _inputs(case, seed):
    """The numbers of a case, on the GPU, from the seed alone."""
    gen = _gen(seed)
    kind = case["kind"]
    if kind == "batch":
        return {"faces": [[f.float() for f in _fourier(n, gen)] for n in _boxes(case)]}
    n, h = _size(case)
    if kind == "liquid":
        return {"faces": _solenoidal(n, h, gen), "fraction": _fraction(n, gen)}
    if kind == "frame":
        faces = [f.float() for f in _fourier(n, gen)]
        p = torch.randn((n[2], n[1], n[0]), dtype=torch.float64, generator=gen, device="cuda")
        return {"faces": faces, "tracer": _blob(n, gen), "fraction": _fraction(n, gen), "pressure": p}
    faces = _fourier(n, gen)
    if kind == "solve":
        return {"rhs": _rhs_of(faces, h, 0.25 * min(h))}
    if kind == "box_flux":
        speed = 0.25 + 0.5 * float(torch.rand((), generator=gen, device="cuda"))
        return {"faces": [f.float() for f in faces], "speed": float(torch.tensor(speed, dtype=torch.float32))}
    dtype = torch.float32 if case.get("storage") == "f32" or case.get("dtype") == "float32" else torch.float64
    out = {"faces": [f.to(dtype) for f in faces]}
    if case.get("tracer"):
        out["tracer"] = _blob(n, gen)
    return out


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    kind = case["kind"]
    torch.cuda.synchronize()  # the library's own streams read these inputs
    if kind == "batch":
        boxes = _boxes(case)
        batch = R.BatchedCarriers([R.GridGeometry(n) for n in boxes], R.CarrierConfig.mixed(pressure=_settings(1e-8)))
        for i, f in enumerate(s["faces"]):
            batch.upload_ptrs(i, *[x.data_ptr() for x in f])
        sizes = [sum(x.numel() for x in f) for f in s["faces"]]
        s["out"] = torch.empty(sum(sizes), dtype=torch.float32, device="cuda")
        s["at"], at = [], 0
        for f in s["faces"]:
            p = []
            for x in f:
                p.append(s["out"].data_ptr() + 4 * at)
                at += x.numel()
            s["at"].append(p)
        s["batch"], s["params"] = batch, R.StepParams(MAXF, cfl=0.5)
        return s
    n, h = _size(case)
    grid = s["grid"] = R.GridGeometry(n, h)
    cells = (n[2], n[1], n[0])
    if kind == "rhs":
        s["operator"] = R.PressureOperator(grid, 1.0)
        s["out"] = torch.empty(cells, dtype=torch.float64, device="cuda")
    elif kind == "advect":
        s["out"] = _blank(n, s["faces"][0].dtype)
    elif kind == "liquid":
        s["state"] = L.LiquidVolumeState(grid, 800.0, (41, 0), s["fraction"])
        s["inlet"] = L.LiquidInlet((4, 0), [[0.0, 0.0]] * 3)
        s["limits"] = L.LiquidVolumeSettings(1.0, 1e-2)
        s["dt"] = _liquid_dt(s["faces"], h)
        s["out"] = torch.empty(cells, dtype=torch.float64, device="cuda")
    elif kind == "frame":
        s["encoder"] = D.Dense3dEncoder(grid)
        s["fields"] = D.Dense3dFields.from_tensors(*s["faces"], s["tracer"], s["fraction"], s["pressure"])
        s["info"] = D.Dense3dFrameInfo(carrier_stamp=(1, 0), liquid_stamp=(2, 0))
        s["out"] = torch.zeros(s["encoder"].bound(), dtype=torch.uint8, device="cuda")
    elif kind == "solve":
        s["operator"] = R.PressureOperator(grid, 1.0)
        s["workspace"] = R.PressureWorkspace(grid, 1 << 62, METHODS[case["method"]])
        s["out"] = torch.empty(cells, dtype=torch.float64, device="cuda")
    elif kind == "box_flux":
        s["workspace"] = B.BoxFluxWorkspace(grid, 1.0, 1 << 62, METHODS[case["method"]])
        v = s["speed"]
        s["boundary"] = B.PrescribedBoxFlux(B.BoxFluxStamp(1, 1), [[-v, v], [0.0, 0.0], [0.0, 0.0]])
        s["settings"] = B.BoxFluxSettings(_settings(1e-8), MAXF)
        s["out"] = _blank(n, torch.float32)
    else:
        sim = R.CarrierSimulation(grid, _config(case))
        sim.upload_ptrs(*[f.data_ptr() for f in s["faces"]], s["tracer"].data_ptr() if case["tracer"] else 0)
        s["sim"] = sim
        s["params"] = R.StepParams(MAXF, cfl=0.5, buoyancy=1.0 if case["tracer"] else 0.0)
        s["out"] = _blank(n, s["faces"][0].dtype)
        if case["tracer"]:
            s["out"].append(torch.empty(cells, dtype=torch.float32, device="cuda"))
    return s


class _View:
    """An f64 device array that the library owns, for a copy out of it (it lives as long as its owner)."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (ptr, False), "version": 2}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "batch":
        for _ in range(case["steps"]):
            for status, _report in s["batch"].step(s["params"]):
                if status:
                    raise RuntimeError(R.status_name(status))
        for i, p in enumerate(s["at"]):
            s["batch"].download_ptrs(i, *p)
        return s["out"]
    if kind == "rhs":
        s["operator"].build_rhs(s["faces"], 0.25, s["out"])
        return s["out"]
    if kind == "advect":
        R.advect_velocity(s["grid"], s["faces"], 0.25 * min(s["grid"].spacing), s["out"])
        return s["out"]
    if kind == "liquid":
        st = s["state"]
        stream = torch.cuda.current_stream().cuda_stream
        st.advance(s["faces"], st.time, s["dt"], (43, 1), s["inlet"], s["limits"], stream=stream)
        return s["out"].copy_(torch.as_tensor(_View(st.fraction_device_ptr(), s["out"].shape), device="cuda"))
    if kind == "frame":
        stream = torch.cuda.current_stream().cuda_stream
        length = s["encoder"].encode_into(s["info"], s["fields"], s["out"].data_ptr(), s["out"].numel(), stream)
        return {"line": s["out"], "length": length}
    if kind == "solve":
        ws = s["workspace"]
        ws.solve_rhs(s["operator"], s["rhs"], 0.25, _settings(case["rel"]))
        return s["out"].copy_(torch.as_tensor(_View(ws.pressure_device_ptr(), s["out"].shape), device="cuda"))
    if kind == "box_flux":
        s["workspace"].project(s["faces"], 0.25 * min(s["grid"].spacing), s["boundary"], s["settings"], s["out"])
        return s["out"]
    s["sim"].step(s["params"])
    s["sim"].download_ptrs(*[o.data_ptr() for o in s["out"]])
    return s["out"]


def work(case):
    kind = case["kind"]
    if kind == "batch":
        boxes = _boxes(case)
        f = sum(3 * (n[0] + 1) * n[1] * n[2] for n in boxes)
        c = sum(n[0] * n[1] * n[2] for n in boxes)
        # every step: the faces read and written, the pressure written; the largest part of the
        # arithmetic is the advection's (three samples of eight corners a face)
        return {"bytes": case["steps"] * (8.0 * f + 8.0 * c), "flops": case["steps"] * 200.0 * f}
    n, _ = _size(case)
    c = n[0] * n[1] * n[2]
    f = sum(math.prod(_face_shape(n, a)) for a in range(3))
    elem = 4 if "float32" in (case.get("dtype"),) or case.get("storage") == "f32" else 8
    if kind == "rhs":
        return {"bytes": elem * f + 8.0 * c, "flops": 9.0 * c}
    if kind == "advect":
        return {"bytes": 2.0 * elem * f, "flops": 200.0 * f}
    if kind == "liquid":
        return {"bytes": 4.0 * f + 16.0 * c, "flops": 60.0 * c}
    if kind == "frame":
        # f32 values of about 16 characters, f64 values of about 24
        return {"bytes": (4.0 + 16.0) * (f + c) + (8.0 + 24.0) * 2 * c, "flops": 0.0}
    if kind == "solve":
        return {"bytes": 16.0 * c, "flops": 30.0 * c}
    if kind == "box_flux":
        return {"bytes": 8.0 * f + 8.0 * c, "flops": 60.0 * c}
    extra = 8.0 * c if case["tracer"] else 0.0
    return {"bytes": 2.0 * elem * f + 8.0 * c + extra, "flops": 200.0 * (f + (c if case["tracer"] else 0))}


# ------------------------------------------------------------------ 64-bit values
def _sample(values, off, xh):
    """Clamped trilinear samples of a [k][j][i] array at scaled positions."""
    dims = values.shape[::-1]
    lo, hi, t = [], [], []
    for d in range(3):
        q = torch.clamp(xh[d] - off[d], 0.0, float(dims[d] - 1))
        f = torch.floor(q)
        lo.append(f.long())
        hi.append(torch.clamp(f.long() + 1, max=dims[d] - 1))
        t.append(q - f)
    flat = values.reshape(-1)
    out = 0.0
    for z in (0, 1):
        for y in (0, 1):
            for x in (0, 1):
                i = (lo[0], hi[0])[x] + dims[0] * ((lo[1], hi[1])[y] + dims[1] * (lo[2], hi[2])[z])
                wt = (t[0] if x else 1 - t[0]) * (t[1] if y else 1 - t[1]) * (t[2] if z else 1 - t[2])
                out = out + wt * flat[i].double()
    return out


def _departure(faces, n, h, pos, dt):
    """Midpoint departure points of the positions, clamped to the box."""
    def velocity(p):
        xh = [p[d] / h[d] for d in range(3)]
        return [_sample(faces[a], [0.0 if d == a else 0.5 for d in range(3)], xh) for a in range(3)]

    def back(v, t):
        return [torch.clamp(pos[d] - t * v[d], 0.0, n[d] * h[d]) for d in range(3)]

    return back(velocity(back(velocity(pos), 0.5 * dt)), dt)


def _positions(shape, off, h, k0, k1):
    pos = []
    for d in range(3):
        x = torch.arange(shape[2 - d], dtype=torch.float64, device="cuda")
        if d == 2:
            x = x[k0:k1]
        view = [1, 1, 1]
        view[2 - d] = -1
        pos.append(((x + off[d]) * h[d]).reshape(view).expand(k1 - k0, shape[1], shape[2]))
    return pos


def _advected(values, off, faces, n, h, dt):
    """A field of the given lattice sampled at its departure points, in slabs of planes."""
    shape = list(values.shape)
    out = torch.empty(shape, dtype=torch.float64, device="cuda")
    slab = max(1, (1 << 22) // (shape[1] * shape[2]))
    for k0 in range(0, shape[0], slab):
        k1 = min(shape[0], k0 + slab)
        dep = _departure(faces, n, h, _positions(shape, off, h, k0, k1), dt)
        out[k0:k1] = _sample(values, off, [dep[d] / h[d] for d in range(3)])
    return out


def _advect_faces(faces, n, h, dt):
    out = []
    for a in range(3):
        f = _advected(faces[a], [0.0 if d == a else 0.5 for d in range(3)], faces, n, h, dt)
        f.select(2 - a, 0).zero_()
        f.select(2 - a, n[a]).zero_()
        out.append(f)
    return out


def _poisson(b, h):
    """The pressure of a sealed box with p[0] = 0: cosine transforms of the 7-point operator."""
    n = b.shape[::-1]
    area = (h[1] * h[2], h[0] * h[2], h[0] * h[1])
    mats, lam = [], 0.0
    for d in range(3):
        m = n[d]
        q = torch.arange(m, dtype=torch.float64, device="cuda")
        c = torch.cos(math.pi * q[:, None] * (2 * q[None, :] + 1) / (2 * m)) * math.sqrt(2.0 / m)
        c[0] *= math.sqrt(0.5)
        mats.append(c)
        view = [1, 1, 1]
        view[2 - d] = -1
        lam = lam + (area[d] / h[d] * 4 * torch.sin(math.pi * q / (2 * m)) ** 2).reshape(view)

    def apply(x, c, d):
        if d == 0:
            return torch.matmul(x, c.T)
        if d == 1:
            return torch.matmul(c, x)
        return torch.matmul(c, x.reshape(x.shape[0], -1)).reshape(c.shape[0], x.shape[1], x.shape[2])

    x = b
    for d in range(3):
        x = apply(x, mats[d], d)
    lam = lam.clone()
    lam[0, 0, 0] = 1.0
    x = x / lam
    x[0, 0, 0] = 0.0
    for d in range(3):
        x = apply(x, mats[d].T, d)
    return x - x[0, 0, 0]


def _correct(faces, p, h, dt):
    """faces less dt grad p on the interior faces (density 1), f64."""
    out = []
    for a in range(3):
        f = faces[a].double().clone()
        m = p.shape[2 - a]
        g = (p.narrow(2 - a, 1, m - 1) - p.narrow(2 - a, 0, m - 1)) / h[a]
        f.narrow(2 - a, 1, m - 1).sub_(dt * g)
        out.append(f)
    return out


def _step_exact(faces, n, h, tracer, buoyancy):
    """One step at CFL 0.5 in 64 bits: (faces, tracer)."""
    faces = [f.double() for f in faces]
    dt = 0.5 / sum(float(faces[a].abs().max()) / h[a] for a in range(3))
    adv = _advect_faces(faces, n, h, dt)
    if tracer is not None and buoyancy:
        m = n[1]
        adv[1].narrow(1, 1, m - 1).add_(dt * buoyancy * 0.5 * (tracer.double().narrow(1, 0, m - 1)
                                                               + tracer.double().narrow(1, 1, m - 1)))
    new = _correct(adv, _poisson(_rhs_of(adv, h, dt), h), h, dt)
    if tracer is not None:
        tracer = _advected(tracer.double(), [0.5] * 3, new, n, h, dt)
    return new, tracer


def _liquid_dt(faces, h):
    """Half the outward Courant limit of the flow."""
    return 0.25 / sum(2.0 * float(faces[a].abs().max()) / h[a] for a in range(3))


def _liquid_exact(f, faces, n, h, dt):
    """One upwind interval of the sealed box in f64."""
    area = (h[1] * h[2], h[0] * h[2], h[0] * h[1])
    volume = h[0] * h[1] * h[2]
    new = f.clone()
    for a in range(3):
        m, ax = n[a], 2 - a
        u = faces[a].double().narrow(ax, 1, m - 1)
        lo, hi = f.narrow(ax, 0, m - 1), f.narrow(ax, 1, m - 1)
        moved = torch.where(u > 0, lo, hi) * u * (dt * area[a] / volume)
        new.narrow(ax, 0, m - 1).sub_(moved)
        new.narrow(ax, 1, m - 1).add_(moved)
    return new


def exact(case, seed):
    kind = case["kind"]
    if kind == "frame":
        return None  # bytes
    s = _inputs(case, seed)
    if kind == "batch":
        out = []
        for n, f in zip(_boxes(case), s["faces"]):
            for _ in range(case["steps"]):
                f = _step_exact(f, n, (1.0, 1.0, 1.0), None, 0.0)[0]
            out += [x.reshape(-1) for x in f]
        return torch.cat(out)
    n, h = _size(case)
    if kind == "rhs":
        return _rhs_of(s["faces"], h, 0.25)
    if kind == "advect":
        return _advect_faces([f.double() for f in s["faces"]], n, h, 0.25 * min(h))
    if kind == "liquid":
        return _liquid_exact(s["fraction"], s["faces"], n, h, _liquid_dt(s["faces"], h))
    if kind == "solve":
        return _poisson(s["rhs"], h)
    if kind == "box_flux":
        f = [x.double() for x in s["faces"]]
        f[0].select(2, 0).fill_(s["speed"])
        f[0].select(2, n[0]).fill_(s["speed"])
        dt = 0.25 * min(h)
        return _correct(f, _poisson(_rhs_of(f, h, dt), h), h, dt)
    faces, tracer = _step_exact(s["faces"], n, h, s.get("tracer"), 1.0)
    return faces + ([tracer] if tracer is not None else [])
