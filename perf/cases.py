"""Workloads of the time-domain acoustic engine, timed through its public entry points.

Each case is one call (or one step of a loop) that a seismic modelling or inversion
program makes again and again: single leapfrog steps on solver data, forward modelling,
misfit gradients and linearised (Born) modelling, in one to three dimensions, FP32 and
FP64, orders 2 to 8, from a grid of a few thousand cells to the full 2D batch and the full
3D volume of the benchmark configurations.  Records are shorter than production records
(the cost of a time step does not depend on its number), but long enough for the source
pulse to enter the model.

``exact`` restates every case in FP64 with plain torch operations.
"""
import math

import numpy as np
import torch

DX = 10.0             # grid spacing in metres, all axes
VMIN, VMAX = 1500.0, 4500.0
CFL = {1: 0.5, 2: 0.4, 3: 0.35}
FREQ = VMIN / (6 * DX)  # six points per shortest wavelength
L2 = 126e6            # wavefields of a pass that fit here need not move to memory every step


def listed():
    return [
        # one step of the drop-in interface (time_step + compute_dWaveOp) on the small survey
        # grid: what a script that inspects wavefields step by step calls, latency only
        dict(name="step-2d-small-f64", kind="step", dim=2, nx=121, ny=1, nz=61, pml=10, order=4, dtype="f64"),
        # the same on a 3D volume, in the solver's default precision
        dict(name="step-3d-f64", kind="step", dim=3, nx=161, ny=161, nz=121, pml=16, order=4, dtype="f64"),
        # a well-log sized 1D inversion: hundreds of tiny steps
        dict(name="gradient-1d-f64", kind="gradient", dim=1, nx=1, ny=1, nz=751, pml=24, order=4, dtype="f64",
             shots=1, receivers=3, steps=800, schedule="checkpoint", checkpoint=0, uneven=False),
        # the small survey (121 x 61 nodes, order 4, one shot, 121 receivers, default precision):
        # the case every user of the package starts with
        dict(name="gradient-2d-small-f64", kind="gradient", dim=2, nx=121, ny=1, nz=61, pml=10, order=4, dtype="f64",
             shots=1, receivers=121, steps=360, schedule="checkpoint", checkpoint=0, uneven=False),
        # modelling one shot on the full 2D grid: quality control of a model, one record at a time
        dict(name="forward-2d-shot-f32", kind="forward", dim=2, nx=1152, ny=1, nz=384, pml=40, order=8, dtype="f32",
             shots=1, receivers=1152, steps=400),
        # modelling in default precision, a few shots on a medium, ragged grid (line searches, reference data)
        dict(name="forward-2d-f64", kind="forward", dim=2, nx=421, ny=1, nz=163, pml=20, order=8, dtype="f64",
             shots=6, receivers=421, steps=150),
        # Born modelling of a shot batch on the coarse grid of a multiscale inversion
        dict(name="born-2d-f32", kind="born", dim=2, nx=289, ny=1, nz=97, pml=10, order=4, dtype="f32",
             shots=16, receivers=289, steps=200),
        # the middle grid of a multiscale batch, records of uneven length, dWaveOp kept in memory
        dict(name="gradient-2d-kept-f32", kind="gradient", dim=2, nx=577, ny=1, nz=193, pml=20, order=6, dtype="f32",
             shots=21, receivers=577, steps=200, schedule="store", checkpoint=64, uneven=True),
        # the full 2D batch: 64 shots through autograd, checkpoints every 64 steps, observed data on the host
        dict(name="gradient-2d-batch-f32", kind="gradient", dim=2, nx=1152, ny=1, nz=384, pml=40, order=8, dtype="f32",
             shots=64, receivers=1152, steps=96, schedule="checkpoint", checkpoint=64, uneven=False),
        # a small 3D inversion in default precision
        dict(name="gradient-3d-small-f64", kind="gradient", dim=3, nx=41, ny=37, nz=33, pml=6, order=4, dtype="f64",
             shots=2, receivers=64, steps=60, schedule="checkpoint", checkpoint=0, uneven=False),
        # 3D modelling of a few shots on a ragged medium volume
        dict(name="forward-3d-f32", kind="forward", dim=3, nx=101, ny=87, nz=75, pml=10, order=4, dtype="f32",
             shots=4, receivers=400, steps=100),
        # the full 3D volume, one shot at a time, 100 x 100 receivers
        dict(name="gradient-3d-f32", kind="gradient", dim=3, nx=400, ny=400, nz=300, pml=20, order=8, dtype="f32",
             shots=1, receivers=10000, steps=40, schedule="checkpoint", checkpoint=20, uneven=False),
    ]


# ---- drawn cases -------------------------------------------------------------------------
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(c):
    """Cell updates of a pass, FP64 ones counted eight times (this chip's FP64 rate is low)."""
    n = _cells(c) * c.get("shots", 1) * c.get("steps", 1)
    n *= {"step": 1, "forward": 1, "born": 2, "gradient": 3}[c["kind"]]
    return n * (8 if c["dtype"] == "f64" else 1) * (3 if c["dim"] == 3 else 1)


_MOST = 6e9  # about the largest listed cases


def draw(rng):
    while True:
        kind = rng.choice(["step", "forward", "forward", "born", "gradient", "gradient", "gradient"])
        dim = rng.choice([2, 3]) if kind == "step" else rng.choice([1, 2, 2, 2, 3, 3])
        c = dict(kind=kind, dim=dim, order=rng.choice([2, 4, 6, 8]), dtype=rng.choice(["f32", "f32", "f64"]),
                 nx=1, ny=1)
        if dim == 1:
            c.update(nz=_log(rng, 150, 2000), pml=_log(rng, 10, 40))
        elif dim == 2:
            c.update(nx=_log(rng, 61, 1152), nz=_log(rng, 45, 384), pml=_log(rng, 8, 40))
        else:
            c.update(nx=_log(rng, 30, 400), ny=_log(rng, 30, 400), nz=_log(rng, 28, 300), pml=_log(rng, 5, 20))
        if kind == "step":
            if _cells(c) > 2e7:
                continue
            return c
        c.update(steps=_log(rng, 40, 400), shots=_log(rng, 1, 4 if dim == 3 else 64))
        if dim == 1:
            c["shots"] = _log(rng, 1, 8)
        c["receivers"] = 3 if dim == 1 else _log(rng, min(24, c["nx"]), c["nx"]) if dim == 2 \
            else _log(rng, 4, min(100, c["nx"], c["ny"])) ** 2
        if kind == "gradient":
            c.update(schedule=rng.choice(["checkpoint", "store"]), checkpoint=rng.choice([0, 64]),
                     uneven=rng.random() < 0.25 and c["dtype"] == "f32")
        if _cost(c) > _MOST:
            continue
        if kind == "gradient" and c["schedule"] == "store" and \
                _cells(c) * c["shots"] * c["steps"] * _bytes(c) > 30e9:
            continue
        return c


# ---- geometry shared by the program's calls and the exact values --------------------------
def _axes(c):
    return [c["nz"]] if c["dim"] == 1 else [c["nx"], c["nz"]] if c["dim"] == 2 else [c["nx"], c["ny"], c["nz"]]


def _padded(c):
    return [n + 2 * c["pml"] for n in _axes(c)]


def _cells(c):
    return math.prod(_padded(c))


def _bytes(c):
    return 8 if c["dtype"] == "f64" else 4


def _pml_amplitude(c):
    return 3 * VMAX * math.log(1e3) / (2 * c["pml"] * DX)


def _model(c, seed):
    """Velocity on the grid: a gradient with depth and smooth lateral perturbations (a start model)."""
    rng = np.random.default_rng(seed)
    n = _axes(c)
    x = np.meshgrid(*[np.linspace(0.0, 1.0, m) for m in n], indexing="ij", sparse=True)
    C = VMIN + (0.9 * VMAX - VMIN) * x[-1]
    p = 0.0
    for _ in range(6):
        arg = rng.uniform(0, 2 * np.pi)
        for a in x:
            arg = arg + 2 * np.pi * rng.uniform(0.5, 4.0) * a
        p = p + np.sin(arg)
    C = np.clip(C * (1.0 + 0.05 * p / 3.0), VMIN, VMAX)
    C.flat[-1] = VMAX  # the time step follows from the largest velocity
    return C.astype(np.float32).astype(np.float64)


def _time_step(c):
    delta = min((n - 1) * DX / (n - 1) for n in _axes(c))
    return CFL[c["dim"]] * delta / VMAX


def _positions(c):
    """(source positions, receiver positions) of the survey: sources spread over the surface,
    receivers the same for every shot; 1D: a source and receivers down the line."""
    ext = [(n - 1) * DX for n in _axes(c)]
    if c["dim"] == 1:
        src = [(ext[0] * 0.2 * (i + 1) / c["shots"],) for i in range(c["shots"])]
        return src, [(ext[0] * f,) for f in np.linspace(0.1, 0.7, c["receivers"])]
    if c["dim"] == 2:
        src = [(ext[0] * (i + 1) / (c["shots"] + 1.0), 0.0) for i in range(c["shots"])]
        return src, [(float(x), 0.0) for x in np.linspace(0.0, ext[0], c["receivers"])]
    m = math.isqrt(c["receivers"])
    src = [(ext[0] * (i + 1) / (c["shots"] + 1.0), ext[1] * 0.5, 0.0) for i in range(c["shots"])]
    return src, [(float(x), float(y), 0.0) for x in np.linspace(0.0, ext[0], m) for y in np.linspace(0.0, ext[1], m)]


def _ricker(t):
    sigma = 1 / (math.pi * FREQ * math.sqrt(2.0))
    x = (np.asarray(t) - 3 * sigma) / (math.sqrt(2.0) * sigma)
    v = -0.5 * (4 * x * x - 2) * np.exp(-x * x)
    v[np.abs(v) < 1e-6] = 0.0
    return v


def _observed_times(c):
    """Recorded samples: another sampling interval than the solver's, over its record."""
    n = max(2, int(math.ceil(c["steps"] / 0.93)) + 1)
    return np.arange(n) * (0.93 * _time_step(c))


def _observed(c, seed, device):
    """Recorded traces [shots, samples, receivers]: a direct arrival and one reflection (FP64)."""
    rng = np.random.default_rng(seed + 1)
    src, rec = _positions(c)
    s = torch.tensor(np.array(src), dtype=torch.float64, device=device)
    r = torch.tensor(np.array(rec), dtype=torch.float64, device=device)
    off = torch.cdist(s, r)[:, None, :]
    t = torch.tensor(_observed_times(c), dtype=torch.float64, device=device)[None, :, None]
    scale = {1: 5.0 + 0 * off, 2: 0.1 / torch.sqrt(1 + off / DX), 3: 1 / (4 * math.pi * (off + DX))}[c["dim"]]
    sigma = 1 / (math.pi * FREQ * math.sqrt(2.0))
    out = 0
    depth = rng.uniform(20.0, 60.0)
    for amp, path in ((1.0, off), (rng.uniform(0.1, 0.3), torch.sqrt(off ** 2 + 4 * depth ** 2))):
        x = (t - path / VMIN - 3 * sigma) / (math.sqrt(2.0) * sigma)
        out = out + amp * scale * (1 - 2 * x * x) * torch.exp(-x * x)
    return out


def _record_steps(c, seed):
    n = c["steps"]
    return tuple(int(v) for v in np.random.default_rng(seed + 2).integers(max(1, n // 2), n + 1, size=c["shots"]))


def _perturbation(c, seed):
    """A smooth model perturbation in squared slowness, about 1 %."""
    rng = np.random.default_rng(seed + 3)
    x = np.meshgrid(*[np.linspace(0.0, 1.0, m) for m in _axes(c)], indexing="ij", sparse=True)
    p = 0.0
    for _ in range(4):
        arg = rng.uniform(0, 2 * np.pi)
        for a in x:
            arg = arg + 2 * np.pi * rng.uniform(1.0, 5.0) * a
        p = p + np.sin(arg)
    return (0.01 * p / 4.0) * _model(c, seed) ** -2


def _step_fields(c, seed, device):
    """(u_{k-1}, {aux name: field}, u_k, rhs) of one step on the padded grid (FP64): smooth
    wavefields, PML state in the padding (psi everywhere in 3D), zero on the outer ring."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    n = _padded(c)
    x = [torch.linspace(0, 1, m, dtype=torch.float64, device=device) for m in n]
    grids = torch.meshgrid(*x, indexing="ij")
    ring = torch.zeros(n, dtype=torch.float64, device=device)
    ring[tuple(slice(1, -1) for _ in n)] = 1.0
    pad = torch.ones(n, dtype=torch.float64, device=device)
    pad[tuple(slice(c["pml"], -c["pml"]) for _ in n)] = 0.0

    def field(scale):
        out = torch.zeros(n, dtype=torch.float64, device=device)
        for _ in range(3):
            k = torch.rand(len(n) + 1, generator=g, dtype=torch.float64)
            arg = 6.28 * float(k[-1])
            for a, gr in enumerate(grids):
                arg = arg + 6.28 * (1 + float(k[a]) * n[a] / 8) * gr
            out += torch.sin(arg)
        return scale * out * ring

    uk = field(1.0)
    um = (uk + field(0.05)) * ring
    aux = {}
    for a in ["z"] if c["dim"] == 1 else ["x", "z"] if c["dim"] == 2 else ["x", "y", "z"]:
        aux["Phi" + a] = field(0.02) * pad
    if c["dim"] == 3:
        aux["psi"] = field(1e-3)
    rhs = field(1e-3)
    if c["dtype"] == "f32":
        um, uk, rhs = um.float().double(), uk.float().double(), rhs.float().double()
        aux = {k: v.float().double() for k, v in aux.items()}
    return um, aux, uk, rhs


# ---- the program's side --------------------------------------------------------------------
def prepare(case, seed):
    import pysit_gb300 as ps
    from pysit_gb300.autograd import FWIMisfit
    from pysit_gb300.engine import WavePlan
    c = dict(case)
    pml = ps.PML(c["pml"] * DX, _pml_amplitude(c))
    domain = ps.RectangularDomain(*[(0.0, (n - 1) * DX, pml, pml) for n in _axes(c)])
    mesh = ps.CartesianMesh(domain, *_axes(c))
    C = _model(c, seed)
    steps = c.get("steps", 100)
    kw = {}
    if c["kind"] != "step":
        kw = dict(checkpoint_every=c.get("checkpoint") or None, gradient_schedule=c.get("schedule", "checkpoint"))
        if c["dim"] == 3:
            kw["pml_psi"] = "consistent"
    solver = ps.ConstantDensityAcousticWave(
        mesh, spatial_accuracy_order=c["order"], trange=(0.0, (steps - 0.5) * _time_step(c)),
        kernel_implementation="cuda", precision="double" if c["dtype"] == "f64" else "single",
        cfl_safety=CFL[c["dim"]], **kw)
    m0 = solver.ModelParameters(mesh, {"C": C.reshape(-1, 1)})
    state = dict(case=c, solver=solver, m0=m0)
    if c["kind"] == "step":
        solver.model_parameters = m0
        um, aux, uk, rhs = _step_fields(c, seed, "cuda")
        sd = solver.DeviceSolverData()
        sd.km1.u[:] = um.reshape(-1, 1)
        sd.k.u[:] = uk.reshape(-1, 1)
        for name, v in aux.items():
            getattr(sd.k, name)[:] = v.reshape(-1, 1)
        state.update(data=sd, rhs=rhs.reshape(-1, 1).to(sd.k.u.dtype))
        return state
    wavelet = ps.RickerWavelet(FREQ, shift_deviations=3)
    src, rec = _positions(c)
    points = [ps.PointReceiver(mesh, p) for p in rec]
    shots = [ps.Shot(ps.PointSource(mesh, p, wavelet), ps.ReceiverSet(mesh, points)) for p in src]
    state["shots"] = shots
    if c["kind"] == "forward":
        solver.model_parameters = m0
        state["plan"] = WavePlan(solver, shots, forward_only=True)
    elif c["kind"] == "born":
        solver.model_parameters = m0
        state["plan"] = WavePlan(solver, shots)
        state["m1"] = torch.tensor(_perturbation(c, seed).reshape(-1), device="cuda")
    elif c["dtype"] == "f64":
        obs = _observed(c, seed, "cuda").cpu().numpy()
        ts = _observed_times(c)
        for s, d in zip(shots, obs):
            s.receivers.ts = ts
            s.receivers.data = d.copy()
        state["objective"] = ps.TemporalLeastSquares(solver)
    else:
        obs = _observed(c, seed, "cuda").float().cpu().pin_memory()
        kw = dict(record_steps=_record_steps(c, seed)) if c["uneven"] else {}
        state["objective"] = FWIMisfit(solver, shots, obs, _observed_times(c), **kw)
        state["C"] = torch.tensor(C, dtype=torch.float32, device="cuda", requires_grad=True)
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "step":
        sd, solver = state["data"], state["solver"]
        solver.time_step(sd, state["rhs"])
        return {"kp1": sd.kp1.data, "dwaveop": solver.compute_dWaveOp("time", sd)}
    if kind == "forward":
        return {"traces": state["plan"].forward()}
    if kind == "born":
        return {"traces": state["plan"].born(state["m1"])}
    if state["case"]["dtype"] == "f64":
        aux = {"objective_value": (True, None)}
        g = state["objective"].compute_gradient(state["shots"], state["m0"], aux_info=aux)
        return {"misfit": float(aux["objective_value"][1]), "gradient": g.data}
    J = state["objective"](state["C"])
    (g,) = torch.autograd.grad(J, state["C"])
    return {"misfit": J.detach(), "gradient": g}


# ---- least work ------------------------------------------------------------------------------
def work(case):
    c = case
    w, cells = _bytes(c), _cells(c)
    R = c["order"] // 2
    per_cell = c["dim"] * 3 * R + 8  # adds and multiply-adds of the symmetric stencil, the leapfrog update
    if c["kind"] == "step":
        aux = {1: 1, 2: 2, 3: 4}[c["dim"]]
        pad = cells - math.prod(_axes(c))
        # u_{k-1}, u_k, C, rhs in, u_{k+1} and dWaveOp out; PML state in and out where it lives
        return {"bytes": float(w * (6 * cells + 2 * aux * pad)), "flops": float(cells * (per_cell + 5))}
    shots, steps = c["shots"], c["steps"]
    traces = shots * steps * c["receivers"] * w
    field = cells * w
    sweeps = {"forward": 1, "born": 2, "gradient": 2}[c["kind"]]
    flops = float(cells) * shots * steps * sweeps * per_cell
    io = traces + 8 * math.prod(_axes(c)) * (1 if c["kind"] == "forward" else 2)
    resident = 3 * field * shots * sweeps + field
    if resident <= L2:
        return {"bytes": float(io), "flops": flops}
    # u_{k-1}, u_k in and u_{k+1} out of every shot and C^2 once, every step; a gradient also
    # writes and reads dWaveOp and updates the image; Born modelling reads m1
    per_step = {"forward": 3 * shots + 1, "born": 6 * shots + 2, "gradient": 10 * shots + 2}[c["kind"]]
    return {"bytes": float(io + per_step * steps * field), "flops": flops}


# ---- exact values: plain torch in FP64 ---------------------------------------------------------
_D1 = {1: [0.5], 2: [2 / 3, -1 / 12], 3: [3 / 4, -3 / 20, 1 / 60], 4: [4 / 5, -1 / 5, 4 / 105, -1 / 280]}
_D2 = {1: [-2.0, 1.0], 2: [-5 / 2, 4 / 3, -1 / 12], 3: [-49 / 18, 3 / 2, -3 / 20, 1 / 90],
       4: [-205 / 72, 8 / 5, -1 / 5, 8 / 315, -1 / 560]}


class _Grid:
    """Padded grid of a case: sigmas, model, stencils (fields are [shots, *grid])."""

    def __init__(self, c, C, device):
        self.c, self.dev = c, device
        self.n = _padded(c)
        self.R = c["order"] // 2
        self.delta = [(n - 1) * DX / (n - 1) for n in _axes(c)]
        self.dt = CFL[c["dim"]] * min(self.delta) / float(np.abs(C).max())
        pad = np.pad(C, [(c["pml"], c["pml"])] * c["dim"], mode="edge")
        self.C2 = torch.tensor(pad, dtype=torch.float64, device=device) ** 2
        prof = _pml_amplitude(c) * np.linspace(0.0, 1.0, c["pml"] + 1) ** 2
        left, right, p = prof[::-1][:-1], prof[1:], c["pml"]
        self.step, self.mesh = [], []  # sigma along each axis: the step's profile and the mesh's map
        for a, n in enumerate(self.n):
            s, m = np.zeros(n), np.zeros(n)
            s[:p], m[:p] = left, left
            m[n - p:] = right
            s[n - p:n - 1] = right[1:]  # the step reads the right profile one node further out
            shape = [1] * c["dim"]
            shape[a] = n
            self.step.append(torch.tensor(s, device=device).reshape(shape))
            self.mesh.append(torch.tensor(m, device=device).reshape(shape))
        self.inner = (slice(None),) + tuple(slice(1, -1) for _ in self.n)

    def sums(self, s):
        d = len(s)
        one = sum(s)
        two = s[0] * s[1] if d == 2 else s[0] * s[1] + s[1] * s[2] + s[2] * s[0] if d == 3 else 0.0
        return one, two, s[0] * s[1] * s[2] if d == 3 else 0.0

    def taps(self, v, a):
        R, n = self.R, self.n[a]
        pad = [0, 0] * (len(self.n) - 1 - a) + [R, R]
        q = torch.nn.functional.pad(v, pad)
        return lambda m: q.narrow(a + 1, R + m, n)

    def d1(self, v, a):
        t = self.taps(v, a)
        return sum(w * (t(m + 1) - t(-m - 1)) for m, w in enumerate(_D1[self.R])) / self.delta[a]

    def d2(self, v, a):
        t = self.taps(v, a)
        w = _D2[self.R]
        return (w[0] * v + sum(w[m] * (t(m) + t(-m)) for m in range(1, self.R + 1))) / self.delta[a] ** 2

    def state(self, shots):
        z = lambda: torch.zeros([shots] + self.n, dtype=torch.float64, device=self.dev)  # noqa: E731
        return {"um": z(), "u": z(), "phi": [z() for _ in self.n], "psi": z() if len(self.n) == 3 else None}

    def advance(self, st, rhs, psi_c2):
        """One step: returns the new state; rhs is a field or None."""
        s, dt, u, um = self.step, self.dt, st["u"], st["um"]
        S1, S2, S3 = self.sums(s)
        F = 0 if rhs is None else rhs
        for a in range(len(self.n)):
            F = F + self.d2(u, a) + self.d1(st["phi"][a], a)
        extra = 0.0
        if len(self.n) == 3:
            extra = S3 * st["psi"]
            if psi_c2:
                F = F - extra
                extra = 0.0
        new = self.C2 * F - extra - (um - 2 * u) / dt ** 2 + S1 * um / (2 * dt) - S2 * u
        new = new * (2 * dt * dt / (2 + dt * S1))
        phi = []
        for a in range(len(self.n)):
            v = st["phi"][a]
            others = S1 - s[a]
            v2 = v - dt * s[a] * v + dt * (others - s[a]) * self.d1(u, a)
            if len(self.n) == 3:
                b, e = [i for i in range(3) if i != a]
                v2 = v2 + dt * s[b] * s[e] * self.d1(st["psi"], a)
            phi.append(self.ringed(v2))
        psi = self.ringed(st["psi"] + dt * u) if len(self.n) == 3 else None
        return {"um": u, "u": self.ringed(new), "phi": phi, "psi": psi}

    def ringed(self, v):
        out = torch.zeros_like(v)
        out[self.inner] = v[self.inner]
        return out

    def dwaveop(self, st, nxt):
        S1, S2, S3 = self.sums(self.mesh)
        um, u, up = st["um"], st["u"], nxt["u"]
        out = (up - 2 * u + um) / self.dt ** 2 + S1 * (up - um) / (2 * self.dt) + S2 * u
        return out + S3 * st["psi"] if len(self.n) == 3 else out

    def points(self, pos):
        """Gaussian taps of points: (padded cells, point, injection weight) as tensors."""
        c = self.c
        cells, which, weight = [], [], []
        sigma = max(self.delta)
        for i, p in enumerate(pos):
            axes = []
            for a, (n, x) in enumerate(zip(_axes(c), p)):
                k = int(round(x / self.delta[a]))
                axes.append(np.arange(max(0, k - 3), min(n, k + 4)))
            idx = np.meshgrid(*axes, indexing="ij")
            r2 = sum((np.linspace(0.0, (n - 1) * DX, n)[k] - x) ** 2 for n, k, x in zip(_axes(c), idx, p))
            w = np.exp(-0.5 * r2 / sigma ** 2) / (math.sqrt(2 * math.pi) * sigma) ** c["dim"]
            flat = np.ravel_multi_index([k + c["pml"] for k in idx], self.n)
            cells.append(flat.ravel())
            which.append(np.full(w.size, i))
            weight.append(w.ravel())
        t = lambda v, d: torch.tensor(np.concatenate(v), dtype=d, device=self.dev)  # noqa: E731
        return t(cells, torch.int64), t(which, torch.int64), t(weight, torch.float64)


def _interpolate(ts, data, new):
    """Linear interpolation of [shots, samples, receivers] along time, zero outside."""
    hi = np.clip(np.searchsorted(ts, new, side="left"), 1, len(ts) - 1)
    f = (new - ts[hi - 1]) / (ts[hi] - ts[hi - 1])
    inside = (new >= ts[0]) & (new <= ts[-1])
    dev = data.device
    hi = torch.tensor(hi, device=dev)
    f = torch.tensor(f, device=dev)[None, :, None]
    m = torch.tensor(inside, device=dev, dtype=torch.float64)[None, :, None]
    y0, y1 = data[:, hi - 1], data[:, hi]
    return ((y1 - y0) * f + y0) * m


def exact(case, seed):
    c = case
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    C = _model(c, seed)
    g = _Grid(c, C, dev)
    if c["kind"] == "step":
        um, aux, uk, rhs = _step_fields(c, seed, dev)
        names = ["z"] if c["dim"] == 1 else ["x", "z"] if c["dim"] == 2 else ["x", "y", "z"]
        st = {"um": um[None], "u": uk[None], "phi": [aux["Phi" + a][None] for a in names],
              "psi": aux["psi"][None] if c["dim"] == 3 else None}
        new = g.advance(st, rhs[None], True)
        parts = [new["u"]] + ([new["psi"]] if c["dim"] == 3 else []) + new["phi"]
        return {"kp1": torch.cat([p.reshape(-1) for p in parts]).reshape(-1, 1),
                "dwaveop": g.dwaveop(st, new).reshape(-1, 1)}
    steps, shots = c["steps"], c["shots"]
    sweeps = {"forward": 1, "born": 2, "gradient": 2}[c["kind"]]
    if _cells(c) * shots * steps * sweeps * (3 if c["dim"] == 3 else 1) > 2.5e10:
        return None  # more than about 20 seconds
    src, rec = _positions(c)
    rc, rr, rw = g.points(rec)
    cell = math.prod(g.delta)
    nrec = len(rec)
    wave = torch.tensor(_ricker(np.arange(steps) * g.dt), dtype=torch.float64, device=dev)
    chunk = max(1, int(64e6 // (8 * _cells(c))))
    traces_all, image, rn2 = [], 0.0, 0.0
    if c["kind"] == "born":
        m1 = torch.tensor(np.pad(_perturbation(c, seed), [(c["pml"], c["pml"])] * c["dim"], mode="edge"), device=dev)
    if c["kind"] == "gradient":
        obs_all = _observed(c, seed, dev)
        if c["dtype"] == "f32":
            obs_all = obs_all.float().double()
        lengths = _record_steps(c, seed) if c["uneven"] else [steps] * shots
    for s0 in range(0, shots, chunk):
        ns = min(chunk, shots - s0)
        sc, sp, sw = g.points(src[s0:s0 + ns])
        sidx = sp * _cells(c) + sc
        shape = [ns] + g.n
        st = g.state(ns)
        lin = g.state(ns) if c["kind"] == "born" else None
        tr = torch.zeros(ns, steps, nrec, dtype=torch.float64, device=dev)
        kept = []
        for k in range(steps):
            u = (lin or st)["u"].reshape(ns, -1)
            tr[:, k].index_add_(1, rr, u[:, rc] * (rw * cell))
            rhs = torch.zeros(ns * _cells(c), dtype=torch.float64, device=dev)
            rhs.index_add_(0, sidx, sw * wave[k])
            nxt = g.advance(st, rhs.reshape(shape), False)
            if c["kind"] == "gradient":
                kept.append(g.dwaveop(st, nxt))
            elif c["kind"] == "born":
                lin = g.advance(lin, -m1 * g.dwaveop(st, nxt), False)
            st = nxt
        if c["kind"] != "gradient":
            traces_all.append(tr)
            continue
        ts = np.arange(steps) * g.dt
        res = _interpolate(_observed_times(c), obs_all[s0:s0 + ns], ts) - tr
        for i in range(ns):
            res[i, lengths[s0 + i]:] = 0.0
        rn2 += float((res * res).sum())
        adj = g.state(ns)
        for k in range(steps - 1, -1, -1):
            image = image + (adj["u"] * kept.pop()).sum(0)
            rhs = torch.zeros(ns, _cells(c), dtype=torch.float64, device=dev)
            rhs.index_add_(1, rc, res[:, k][:, rr] * rw)
            adj = g.advance(adj, rhs.reshape(shape), False)
    if c["kind"] != "gradient":
        return {"traces": torch.cat(traces_all)}
    grad = g.dt * image
    p = c["pml"]
    for a in range(c["dim"]):  # the padding folds onto the boundary nodes
        n = grad.shape[a]
        core = grad.narrow(a, p, n - 2 * p).clone()
        core.narrow(a, 0, 1).add_(grad.narrow(a, 0, p).sum(a, keepdim=True))
        core.narrow(a, n - 2 * p - 1, 1).add_(grad.narrow(a, n - p, p).sum(a, keepdim=True))
        grad = core
    if c["dtype"] == "f64":
        return {"misfit": 0.5 * g.dt * rn2, "gradient": grad.reshape(-1, 1)}
    dC = grad * (-2.0 * cell) * torch.tensor(C, device=dev) ** -3
    return {"misfit": torch.tensor(0.5 * g.dt * rn2, dtype=torch.float64), "gradient": dC}
