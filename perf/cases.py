"""Performance cases of the phase-field step.

Each case is one piece of work that a program hands to the library through
its Python binding (mmsp_gb300.native), which mirrors the C ABI call by call:

``update``   one plugin call on a host grid: create, upload, step, reduce,
             download, destroy (mmsp_gpu_update)
``step``     a handle kept by the program: start state in, a run of steps,
             state out, all on the device (upload_device, step,
             download_device)
``batch``    many independent 2D grids advanced together, host buffers in and
             out (upload_all, step, download_all on pinned memory)
``sparse``   sparse grain growth: host lists in, steps, host lists out
``serve``    a burst of mixed solves through the request loop, submitted,
             awaited and fetched

listed() gives the named cases, draw() more of the same ranges, prepare() the
inputs and handles, run() one pass, work() the bytes and operations of a
pass, exact() the results in 64-bit arithmetic by plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mmsp_gb300 import native

# Time step and coefficients of each model, as its configurations have them.
PARAMS = {
    "ch": dict(kappa=1.0, mobility=1.0),
    "ch_poly": dict(dt=0.01, kappa=1.0, mobility=1.0, r=1.0, u=1.0),
    "ac": dict(dt=0.05, kappa=2.0, mobility=1.0, gamma=1.5),
    "gg": dict(dt=0.01),
    "zener": dict(dt=0.01),
    "ac_poly": dict(dt=0.01, kappa=1.0, mobility=1.0, r=1.0, u=1.0),
    "ostwald": dict(dt=0.001, kappa=2.0, mobility=1.0),
    "ch_convex": {},
}
OSTWALD = dict(D=1.0, Ca=0.05, Cb=0.95, A=2.0, delta=1.0, eps=3.0)
CONVEX = dict(C0=0.45, Ca=0.05, Cb=0.95, A=2.0, omega=1.2, tol=1e-14, D=2.0 / 0.9, K=2.0)
SPARSE_SLOTS = 16


def listed():
    return [
        # The smallest use: update(grid, steps) of a little host grid, as a program that calls the plugin
        # between other work of its own does; set-up, launches and transfers count, not the arithmetic.
        dict(name="update_ch2d_64_f64", kind="update", model="ch", shape="64x64", fields=1, dtype="f64",
             contract=False, dx=1.0, steps=20),
        # The plain 2D Cahn-Hilliard study: 256 x 256, FP64 in the reference's operation order.
        dict(name="ch2d_256_f64", kind="step", model="ch", shape="256x256", fields=1, dtype="f64",
             contract=False, dx=1.0, steps=500),
        # The large plain solve: 256^3 in FP64, contracted form.
        dict(name="ch3d_256_f64_contract", kind="step", model="ch", shape="256x256x256", fields=1, dtype="f64",
             contract=True, dx=1.0, steps=50),
        # The same grid in the precision form.
        dict(name="ch3d_256_f32", kind="step", model="ch", shape="256x256x256", fields=1, dtype="f32",
             contract=False, dx=1.0, steps=200),
        # An odd-sized 3D solve, as served requests have any side.
        dict(name="ch3d_187_f32", kind="step", model="ch", shape="187x187x187", fields=1, dtype="f32",
             contract=False, dx=1.0, steps=200),
        # Grain growth with 8 order parameters in the precision form.
        dict(name="ac3d_128_n8_f32", kind="step", model="ac", shape="128x128x128", fields=8, dtype="f32",
             contract=False, dx=1.0, steps=100),
        # Grain growth on a ragged grid with many order parameters, as served requests have them.
        dict(name="ac3d_74_n14_f32", kind="step", model="ac", shape="74x74x74", fields=14, dtype="f32",
             contract=False, dx=1.0, steps=200),
        # The plain FP64 grain growth that the precision form is compared with.
        dict(name="ac3d_128_n8_f64", kind="step", model="ac", shape="128x128x128", fields=8, dtype="f64",
             contract=False, dx=1.0, steps=10),
        # A parameter study: 256 grids of uneven sizes and coefficients, host to host.
        dict(name="batch_256_f32", kind="batch", count=256, dtype="f32", steps=1000),
        # Sparse grain growth with item lists, host to host.
        dict(name="sparse2d_512", kind="sparse", shape="512x512", grains=160, steps=500),
        # The semi-implicit solve on the example's grid.
        dict(name="convex_400x200", kind="step", model="ch_convex", shape="400x200", fields=2, dtype="f64",
             contract=False, dx=1.0, steps=5),
        # Mixed solves served together: 2D and 3D Cahn-Hilliard and grain growth of any side.
        dict(name="serve_16", kind="serve", requests=16, mix=11),
    ]


# --------------------------------------------------------------------------- drawn cases

def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _steps_within(rng, seconds_per_step, lo, hi, most=0.02):
    """A step count in [lo, hi] (by its logarithm) whose pass stays below about `most` seconds."""
    cap = max(1, int(most / seconds_per_step))
    return max(1, min(cap, _log_int(rng, lo, hi)))


def _step_seconds(case):
    """A rough time of one step, to bound the cost of drawn cases."""
    ops, nbytes = _step_work(case)
    return 4e-6 + (ops / 3e11 if case["dtype"] == "f64" else nbytes / 1.5e12)


def draw(rng):
    kind = rng.choice(["update", "ch2d", "ch3d", "ch3d", "ac3d", "ac3d", "batch", "sparse", "convex", "serve"])
    if kind == "update":
        model = rng.choice(["ch", "ch_poly", "ac", "gg", "zener", "ac_poly", "ostwald"])
        dim = rng.choice([1, 2, 2, 3])
        cells = _log_int(rng, 1 << 8, 1 << 16)
        shape = "x".join(str(max(12, int(round(cells ** (1.0 / dim) * rng.uniform(0.7, 1.4))))) for _ in range(dim))
        fields = 1 if model in ("ch", "ch_poly", "ac_poly") else 3 if model == "zener" else rng.randint(2, 5)
        return dict(kind="update", model=model, shape=shape, fields=fields, dtype=rng.choice(["f64", "f32"]),
                    contract=False, dx=rng.choice([1.0, 1.0, 1.25]), steps=rng.randint(1, 40))
    if kind == "ch2d":
        dtype = rng.choice(["f64", "f64", "f32"])
        case = dict(kind="step", model=rng.choice(["ch", "ch", "ch_poly"]),
                    shape="%dx%d" % (_log_int(rng, 64, 1024), _log_int(rng, 64, 1024)), fields=1, dtype=dtype,
                    contract=dtype == "f64" and rng.random() < 0.4, dx=rng.choice([1.0, 1.0, 1.0, 1.25]))
        case["steps"] = _steps_within(rng, _step_seconds(case), 50, 1000)
        return case
    if kind == "ch3d":
        dtype = rng.choice(["f32", "f32", "f64"])
        n = _log_int(rng, 32, 250)
        sides = [n, n, n] if rng.random() < 0.6 else [_log_int(rng, 32, 250) for _ in range(3)]
        case = dict(kind="step", model=rng.choice(["ch", "ch", "ch_poly"]), shape="x".join(map(str, sides)), fields=1,
                    dtype=dtype, contract=dtype == "f64" and rng.random() < 0.5, dx=rng.choice([1.0, 1.0, 1.0, 1.25]))
        case["steps"] = _steps_within(rng, _step_seconds(case), 20, 400)
        return case
    if kind == "ac3d":
        dtype = rng.choice(["f32", "f32", "f64"])
        n = _log_int(rng, 32, 128)
        sides = [n, n, n] if rng.random() < 0.6 else [_log_int(rng, 32, 128) for _ in range(3)]
        model = rng.choice(["ac", "ac", "ac", "gg"])
        case = dict(kind="step", model=model, shape="x".join(map(str, sides)), fields=rng.randint(4, 16), dtype=dtype,
                    contract=False, dx=rng.choice([1.0, 1.0, 1.0, 1.25]))
        case["steps"] = _steps_within(rng, _step_seconds(case), 10, 400)
        return case
    if kind == "batch":
        count = _log_int(rng, 16, 256)
        dtype = rng.choice(["f32", "f32", "f64"])
        per_step = 5e-6 + count * 1.0e5 * (17 / 3e11 if dtype == "f64" else 1.2e-12)
        return dict(kind="batch", count=count, dtype=dtype, steps=_steps_within(rng, per_step, 100, 1000))
    if kind == "sparse":
        dim = rng.choice([2, 2, 3])
        shape = "x".join(str(_log_int(rng, 128, 500) if dim == 2 else _log_int(rng, 24, 56)) for _ in range(dim))
        # a list holds every grain within about 25 cells: no more grains than keep it within its slots
        cells = math.prod(int(n) for n in shape.split("x"))
        return dict(kind="sparse", shape=shape, grains=rng.randint(8, max(14, cells // 1700) if dim == 2 else 14),
                    steps=_log_int(rng, 50, 500))
    if kind == "convex":
        dim = rng.choice([2, 2, 3])
        shape = "x".join(str(2 * (_log_int(rng, 64, 400) // 2 if dim == 2 else _log_int(rng, 16, 40) // 2))
                         for _ in range(dim))
        return dict(kind="step", model="ch_convex", shape=shape, fields=2, dtype="f64", contract=False, dx=1.0,
                    steps=rng.randint(1, 4))
    case = dict(kind="serve", requests=rng.randint(4, 15), mix=rng.randint(100, 10**6))
    most = work(listed()[-1])
    while case["requests"] > 2 and any(work(case)[k] > most[k] for k in most):
        case["requests"] -= 1   # no heavier than the listed burst
    return case


# --------------------------------------------------------------------------- inputs

def _shape(case):
    return tuple(int(s) for s in case["shape"].split("x"))


def _np_dtype(case):
    return np.float64 if case["dtype"] == "f64" else np.float32


def _torch_dtype(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _rand(shape, gen):
    return torch.rand(shape, generator=gen, dtype=torch.float64, device=gen.device)


def _grains(shape, points, gen):
    """Grain index of every cell of a periodic Voronoi tessellation."""
    dev = gen.device
    seeds = (_rand((points, len(shape)), gen) * torch.tensor(shape, dtype=torch.float64, device=dev)).float().cpu()
    axes = [torch.arange(n, dtype=torch.float32, device=dev) for n in shape]
    best = torch.full(shape, math.inf, dtype=torch.float32, device=dev)
    grain = torch.zeros(shape, dtype=torch.int32, device=dev)
    for p in range(points):
        d2 = None
        for a, n in enumerate(shape):
            d = (axes[a] - float(seeds[p, a])).abs()
            d = torch.minimum(d, n - d) ** 2
            d = d.reshape([-1 if b == a else 1 for b in range(len(shape))])
            d2 = d if d2 is None else d2 + d
        near = d2 < best
        best = torch.where(near, d2, best)
        grain[near] = p
    return grain


def _start(case, seed):
    """The start state in FP64, field-major ([fields] + shape; scalar models: shape)."""
    gen = torch.Generator(device=_device())
    gen.manual_seed(int(seed) * 7919 + 17)
    shape, model, n = _shape(case), case["model"], case["fields"]
    if model == "ch":       # a quench near the middle of the miscibility gap
        mean = 0.4 + 0.1 * float(_rand((1,), gen)[0])
        return mean + 0.02 * (2 * _rand(shape, gen) - 1)
    if model in ("ch_poly", "ac_poly"):
        return 0.2 * (2 * _rand(shape, gen) - 1)
    if model == "ch_convex":
        c = CONVEX["C0"] + 0.25 * _rand(shape, gen) - 0.125
        C0, Ca, Cb, A = CONVEX["C0"], CONVEX["Ca"], CONVEX["Cb"], CONVEX["A"]
        B = A / (Ca - C0) ** 2
        f = -A * (c - C0) + B * (c - C0) ** 3 + Ca * (c - Ca) ** 3 + Cb * (c - Cb) ** 3
        return torch.stack([c, f - CONVEX["K"] * _lap(c, len(shape), 1.0)])
    if model == "ostwald":
        s = 0.1 * _rand((n,) + shape, gen)
        s[0] = _rand(shape, gen)
        s[1] = 1.0 - s[0]
        return s
    # grain growth: one order parameter at 1 in each grain
    grain = _grains(shape, 60, gen) % n
    return torch.stack([(grain == k).double() for k in range(n)])


def _dt(case):
    if case["model"] == "ch":
        return 0.002 if len(_shape(case)) == 3 else 0.005
    return PARAMS[case["model"]].get("dt")


def _desc(case):
    shape, model = _shape(case), case["model"]
    p = dict(PARAMS[model])
    p["dt"] = _dt(case)
    return native.make_desc(shape, case["fields"], _np_dtype(case), model, dx=[case["dx"]] * len(shape),
                            contract=case["contract"], **p)


_STREAM = None


def _program_stream():
    """The one stream on which the program orders its device work."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


class _StepState:
    def __init__(self, case, seed):
        self.steps = case["steps"]
        self.x0 = _start(case, seed).to(_torch_dtype(case)).contiguous()
        self.out = torch.empty_like(self.x0)
        self.nbytes = self.x0.numel() * self.x0.element_size()
        self.stepper = native.Stepper(_desc(case))
        self.stepper.set_stream(_program_stream().cuda_stream)

    def run(self):
        s = self.stepper
        s.upload_device(self.x0.data_ptr(), self.nbytes)
        s.step(self.steps)
        s.download_device(self.out.data_ptr(), self.nbytes)
        return self.out


class _UpdateState:
    def __init__(self, case, seed):
        self.steps = case["steps"]
        x = _start(case, seed)
        if case["fields"] > 1:
            x = x.movedim(0, -1)   # cell-major, as the host grid's vectors lie
        self.host = np.ascontiguousarray(x.cpu().numpy(), dtype=_np_dtype(case))
        self.desc = _desc(case)

    def run(self):
        out, st = native.update(self.host, self.steps, self.desc)
        return [out, st.mass, st.energy]


def _batch_grids(case):
    """(side, kappa, mean) of each grid: sides uniform in 64..512 by 32."""
    rng = np.random.default_rng(case["count"])
    return [(int(32 * rng.integers(2, 17)), float(rng.uniform(0.5, 2.0)), float(rng.uniform(0.3, 0.7)))
            for _ in range(case["count"])]


def _batch_start(case, seed):
    gen = torch.Generator(device=_device())
    gen.manual_seed(int(seed) * 7919 + 17)
    return [(mean + 0.01 * (2 * _rand((n, n), gen) - 1)).to(_torch_dtype(case)) for n, _, mean in _batch_grids(case)]


class _BatchState:
    def __init__(self, case, seed):
        grids, x0 = _batch_grids(case), _batch_start(case, seed)
        total = sum(n * n for n, _, _ in grids)
        self.host = torch.empty(total, dtype=_torch_dtype(case), pin_memory=True)
        self.out = torch.empty(total, dtype=_torch_dtype(case), pin_memory=True)
        self.host.copy_(torch.cat([x.reshape(-1) for x in x0]))
        torch.cuda.synchronize()
        self.src, self.dst, at = [], [], 0
        for n, _, _ in grids:
            self.src.append(self.host[at:at + n * n].numpy().reshape(n, n))
            self.dst.append(self.out[at:at + n * n].numpy().reshape(n, n))
            at += n * n
        self.steps = case["steps"]
        self.batch = native.Batch([native.make_desc((n, n), 1, _np_dtype(case), "ch", dt=0.005, kappa=k, mobility=1.0)
                                   for n, k, _ in grids])
        self.batch.upload_all(self.src)
        self.batch.tune()

    def run(self):
        self.batch.upload_all(self.src)
        self.batch.step(self.steps)
        self.batch.download_all(self.dst)
        return self.out


class _SparseState:
    def __init__(self, case, seed):
        gen = torch.Generator(device=_device())
        gen.manual_seed(int(seed) * 7919 + 17)
        shape = _shape(case)
        grain = _grains(shape, case["grains"], gen).cpu().numpy()
        self.count = np.ones(shape, np.int32)
        self.index = np.zeros(shape + (SPARSE_SLOTS,), np.int32)
        self.value = np.zeros(shape + (SPARSE_SLOTS,), np.float64)
        self.index[..., 0] = grain
        self.value[..., 0] = 1.0
        self.steps = case["steps"]
        self.stepper = native.Stepper(native.make_desc(shape, SPARSE_SLOTS, np.float64, "sparse_gg"))

    def run(self):
        self.stepper.sparse_upload(self.count, self.index, self.value)
        self.stepper.step(self.steps)
        return list(self.stepper.sparse_download())


def _serve_mix(case):
    """The request mix: half 2D Cahn-Hilliard (sides 64-1024), three tenths 3D (sides 32-256), the rest
    grain growth (4-16 order parameters, sides 32-128); 100 to 800 steps."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for i in range(case["requests"]):
        kind = i % 10 / 10.0
        c = dict(dtype="f32", contract=False, dx=1.0, fields=1, steps=int(round(100 * 8 ** rng.random())))
        if kind < 0.5:
            n = int(rng.integers(64, 1025))
            c.update(model="ch", shape="%dx%d" % (n, n))
        elif kind < 0.8:
            n = int(rng.integers(32, 257))
            c.update(model="ch", shape="%dx%dx%d" % (n, n, n))
        else:
            n = int(rng.integers(32, 129))
            c.update(model="ac", shape="%dx%dx%d" % (n, n, n), fields=int(rng.integers(4, 17)))
        out.append(c)
    return out


class _ServeState:
    def __init__(self, case, seed):
        self.requests = []
        for i, c in enumerate(_serve_mix(case)):
            x = _start(c, seed * 64 + i)
            if c["fields"] > 1:
                x = x.movedim(0, -1)
            self.requests.append((_desc(c), np.ascontiguousarray(x.cpu().numpy(), dtype=np.float32), c["steps"]))
        self.server = native.Server(budget_bytes=8 << 30)

    def run(self):
        ids = [self.server.submit(d, x, steps) for d, x, steps in self.requests]
        out = []
        for rid in ids:
            self.server.wait(rid)
            out.append(self.server.fetch(rid))
        return out


_STATES = {"step": _StepState, "update": _UpdateState, "batch": _BatchState, "sparse": _SparseState,
           "serve": _ServeState}


def prepare(case, seed):
    state = _STATES[case["kind"]](case, seed)
    torch.cuda.synchronize()   # the start state is there before another stream reads it
    return state


def run(state):
    return state.run()


# --------------------------------------------------------------------------- work

def _step_work(case):
    """(operations, state bytes in and out) of one step of a dense model, in the reference's expressions."""
    shape, model, n = _shape(case), case["model"], case["fields"]
    cells, dim = math.prod(shape), len(shape)
    lap = 3 * dim - 1
    per_cell = {"ch": 2 * lap + 7, "ch_poly": 2 * lap + 9, "ac": n * (lap + 13), "gg": n * (lap + 12),
                "zener": n * (lap + 12), "ac_poly": lap + 9, "ostwald": 2 * lap + 22 + (n - 1) * (lap + 12),
                # one red-black iteration of the solve (about a hundred run per step)
                "ch_convex": 100 * (2 * lap + 22)}[model]
    return float(cells * per_cell), 2.0 * cells * n * (8 if case["dtype"] == "f64" else 4)


def work(case):
    kind = case["kind"]
    if kind in ("step", "update"):
        ops, nbytes = _step_work(case)
        return {"bytes": nbytes, "flops": ops * case["steps"]}
    if kind == "batch":
        cells = sum(n * n for n, _, _ in _batch_grids(case))
        return {"bytes": 2.0 * cells * (8 if case["dtype"] == "f64" else 4), "flops": 17.0 * cells * case["steps"]}
    if kind == "sparse":
        # lists in and out; at least one item updated per cell and step
        cells, dim = math.prod(_shape(case)), len(_shape(case))
        return {"bytes": 2.0 * cells * (4 + SPARSE_SLOTS * 12), "flops": float(cells) * case["steps"] * (3 * dim + 13)}
    both = [_step_work(c) + (c["steps"],) for c in _serve_mix(case)]
    return {"bytes": sum(b for _, b, _ in both), "flops": sum(o * s for o, _, s in both)}


# --------------------------------------------------------------------------- 64-bit results

def _lap(f, dim, dx):
    """Periodic Laplacian over the last `dim` axes."""
    out = (-2.0 * dim) * f
    for a in range(-dim, 0):
        out += torch.roll(f, 1, a)
        out += torch.roll(f, -1, a)
    return out if dx == 1.0 else out / (dx * dx)


def _ch_run(c, dim, dx, model, dt, kappa, steps):
    for _ in range(steps):
        f = 2 * c * (1 - c) * (1 - 2 * c) if model == "ch" else c ** 3 - c
        c = c + dt * _lap(f - kappa * _lap(c, dim, dx), dim, dx)
    return c


def _ostwald_step(s, dim, dx):
    o, p = OSTWALD, PARAMS["ostwald"]
    C, e = s[0], s[1:]
    Cm = 0.5 * (o["Ca"] + o["Cb"])
    B, g = o["A"] / (o["Cb"] - Cm) ** 2, 2.0 / (o["Cb"] - o["Ca"]) ** 2
    D2 = g / o["delta"] ** 2
    sq = (e * e).sum(0)
    w = -o["A"] * (C - Cm) + B * (C - Cm) ** 3 + D2 * (C - o["Ca"]) ** 3 + D2 * (C - o["Cb"]) ** 3
    w = w - g * (C - o["Ca"]) * sq - p["kappa"] * _lap(C, dim, dx)
    new = torch.empty_like(s)
    new[0] = C + p["dt"] * o["D"] * _lap(w, dim, dx)
    new[1:] = e - p["dt"] * p["mobility"] * (-g * (C - o["Ca"]) ** 2 + o["delta"] * e ** 3
                                             + o["eps"] * e * (sq - e * e) - p["kappa"] * _lap(e, dim, dx))
    return new


def _convex_run(s, dim, steps):
    """Convex splitting by red-black over-relaxation, checked after iterations 1-4 and every 5th."""
    q = CONVEX
    C0, Ca, Cb, A, K, D, om = q["C0"], q["Ca"], q["Cb"], q["A"], q["K"], q["D"], q["omega"]
    dt = 1.0 / (D * K)
    B = A / (Ca - C0) ** 2
    QA, QB = B + Ca + Cb, 3 * (B * C0 + Ca ** 2 + Cb ** 2)
    QC, QD = 3 * (B * C0 ** 2 + Ca ** 3 + Cb ** 3), B * C0 ** 3 + Ca ** 4 + Cb ** 4
    lw = 2.0 * dim
    parity = sum(torch.arange(n, device=s.device).reshape([-1 if b == a else 1 for b in range(dim)])
                 for a, n in enumerate(s.shape[1:])) % 2
    old, guess = s, s.clone()
    for _ in range(steps):
        c0 = old[0]
        expansive = -A * (c0 - C0) - QB * c0 ** 2 - QD
        norm = (c0 ** 2 + expansive ** 2).sum()
        it, res = 0, 1.0
        while it < 10000 and res > q["tol"]:
            for skip in (1, 0):
                c, u = guess[0], guess[1]
                A21 = -(QA * c * c + QC) - K * lw
                det = 1.0 - dt * D * lw * A21
                B1 = c0 + D * dt * (_lap(u, dim, 1.0) + lw * u)
                B2 = expansive - K * (_lap(c, dim, 1.0) + lw * c)
                on = parity != skip
                guess[0] = torch.where(on, om * (B1 - B2 * (dt * D * lw)) / det + (1 - om) * c, c)
                guess[1] = torch.where(on, om * (B2 - B1 * A21) / det + (1 - om) * u, u)
            it += 1
            if it < 5 or it % 5 == 0:
                c, u = guess[0], guess[1]
                r1 = c0 - (c - D * dt * _lap(u, dim, 1.0))
                r2 = expansive - (u - (QA * c ** 3 + QC * c) + K * _lap(c, dim, 1.0))
                res = float(torch.sqrt((r1 ** 2 + r2 ** 2).sum() / norm)) / (2.0 * c.numel())
        old, guess = guess, old.clone()
    return old


def _dense_exact(case, x):
    """The state after the case's steps from the field-major FP64 state x."""
    model, dim, dx, steps = case["model"], len(_shape(case)), case["dx"], case["steps"]
    p = PARAMS[model]
    if model in ("ch", "ch_poly"):
        return _ch_run(x, dim, dx, model, _dt(case), p["kappa"], steps)
    if model == "ch_convex":
        return _convex_run(x, dim, steps)
    for _ in range(steps):
        if model == "ostwald":
            x = _ostwald_step(x, dim, dx)
        elif model == "ac_poly":
            x = x - p["dt"] * (x ** 3 - x - p["kappa"] * _lap(x, dim, dx))
        else:
            lap, sq = _lap(x, dim, dx), (x * x).sum(0)
            if model == "ac":
                e = x * (x * x - 1.0 + 2.0 * p["gamma"] * (sq - x * x)) - p["kappa"] * lap
            else:
                e = 2.0 * (x * sq - lap) - x - x ** 3
            new = x - p["dt"] * e
            if model == "zener":
                new[0] = x[0]   # the particles do not move
            x = new
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "sparse":
        return None   # the lists keep stale items of two steps back: no dense restatement gives them
    if kind == "batch":
        grids = _batch_grids(case)
        x0 = [x.double() for x in _batch_start(case, seed)]
        out = [None] * len(grids)
        for side in sorted({n for n, _, _ in grids}):
            at = [i for i, (n, _, _) in enumerate(grids) if n == side]
            kappa = torch.tensor([grids[i][1] for i in at], dtype=torch.float64, device=x0[0].device).reshape(-1, 1, 1)
            done = _ch_run(torch.stack([x0[i] for i in at]), 2, 1.0, "ch", 0.005, kappa, case["steps"])
            for k, i in enumerate(at):
                out[i] = done[k].reshape(-1)
        return torch.cat(out).cpu()
    if kind == "serve":
        out = []
        for i, c in enumerate(_serve_mix(case)):
            x = _dense_exact(c, _start(c, seed * 64 + i).float().double())
            out.append((x.movedim(0, -1) if c["fields"] > 1 else x).cpu().numpy())
        return out
    x = _start(case, seed).to(_torch_dtype(case)).double()
    x = _dense_exact(case, x)
    if kind == "step":
        return x
    mass = float(x.sum()) * case["dx"] ** len(_shape(case))
    return [(x.movedim(0, -1) if case["fields"] > 1 else x).cpu().numpy(), mass, None]
