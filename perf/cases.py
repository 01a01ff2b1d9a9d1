"""Performance cases of the time-step framework, through its Python entry points.

Most cases are one forecast leg as a program runs it: a host state goes up
(``Model.upload``), the model takes ``steps`` steps (``Model.step``) and the whole state
comes back (``Model.download``), on page-locked host arrays.  The sizes run from the
32 x 32 x 40 bubble to the 1024 x 1024 x 64 moist grid.  Beside them: one step from host
arrays to host arrays (``Model.step_host``, the call of a program that keeps its state on
the host), an ensemble of uneven members, scalar transport on a device array, and the
training of the learned warm rain.

A case with ``tuned`` picks its tiles with ``Model.autotune`` first, as the benchmark
does; one without keeps the library's choice, as the idealized driver does.

``exact`` restates the step in 64 bits with torch tensors: SSPRK3 slow tendencies,
acoustic substeps, tracers and warm rain with fallout, on flat levels and on terrain.
"""
import importlib
import math
import os

import numpy as np
import torch

STATE = ("rho", "rho_theta", "u", "v", "w")
TRACERS = ("qv", "qc", "qr")
RD, P0, KAPPA, RV, LV, GRAVITY = (float(np.float32(x)) for x in (287.05, 1.0e5, 0.2854, 461.5, 2.5e6, 9.81))
FALL_SPEED = 12.0  # m/s, as in the moist benchmark
EXACT_MOST = 1.4e9  # cells x steps x substeps that exact() takes on


def _gwm():
    return importlib.import_module("gpu-wm-next_b200")


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# --------------------------------------------------------------------------------------
# cases
def _leg(name, kind, nx, ny, nz, steps, substeps, dt, spacing, z_top, open_sides=False, tuned=False, surrogate=False):
    return {"name": name, "path": "leg", "kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": steps,
            "substeps": substeps, "dt": dt, "spacing": spacing, "z_top": z_top, "open": open_sides, "tuned": tuned,
            "surrogate": surrogate}


def listed():
    return [
        # the warm bubble of the idealized driver at its own size: latency of small kernels
        _leg("bubble_32x32x40", "bubble", 32, 32, 40, 20, 4, 0.5, 500.0, 10000.0),
        # a ragged dry limited area with open sides: a cold pool on the driver's tiles
        _leg("cold_pool_open_93x61x50", "cold_pool", 93, 61, 50, 20, 3, 0.5, 1000.0, 12500.0, open_sides=True),
        # one moist member of ensemble size
        _leg("moist_128x128x64", "moist", 128, 128, 64, 20, 4, 1.0, 3000.0, 16000.0, tuned=True),
        # an ordinary moist limited area, ragged, open sides
        _leg("moist_open_517x389x50", "moist", 517, 389, 50, 10, 6, 1.0, 3000.0, 16000.0, open_sides=True, tuned=True),
        # the moist benchmark grid: the largest leg
        _leg("moist_1024x1024x64", "moist", 1024, 1024, 64, 20, 6, 1.0, 3000.0, 16000.0, tuned=True),
        # the moist step with the learned warm rain
        _leg("learned_rain_512x512x64", "moist", 512, 512, 64, 10, 6, 1.0, 3000.0, 16000.0, tuned=True, surrogate=True),
        # the mountain wave: terrain, stretched levels, damping layer
        _leg("mountain_512x512x80", "mountain", 512, 512, 80, 10, 6, 0.5, 1000.0, 20000.0, tuned=True),
        # a small moist limited area over terrain on the driver's tiles
        _leg("moist_terrain_open_201x163x40", "moist_mountain", 201, 163, 40, 10, 4, 1.0, 2000.0, 16000.0,
             open_sides=True),
        # uneven members advanced side by side in one context
        {"name": "ensemble_8", "path": "ensemble", "members": 8, "low": 64, "high": 256, "steps": 10, "substeps": 4,
         "dt": 1.0, "tuned": True, "draw": 5},
        # one step of a program that keeps its state on the host
        {"name": "host_step_384x384x64", "path": "host", "kind": "moist", "nx": 384, "ny": 384, "nz": 64, "steps": 1,
         "substeps": 6, "dt": 1.0, "spacing": 3000.0, "z_top": 16000.0, "open": False, "tuned": True,
         "surrogate": False},
        # passive transport of one field on the device
        {"name": "scalar_256x256x64", "path": "scalar", "nx": 256, "ny": 256, "nz": 64, "steps": 30, "open": False},
        # training of the learned warm rain: forward, backward and Adam
        {"name": "train_131072", "path": "train", "samples": 131072, "batch": 16384, "epochs": 1},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case: sizes over their logarithm, odd ones among them, any of the paths."""
    path = rng.choice(["leg"] * 6 + ["host", "scalar", "train", "ensemble"])
    if path == "scalar":
        return {"path": path, "nx": _log_int(rng, 33, 512), "ny": _log_int(rng, 33, 512), "nz": rng.randint(16, 80),
                "steps": rng.randint(5, 40), "open": rng.random() < 0.5}
    if path == "train":
        return {"path": path, "samples": _log_int(rng, 1 << 15, 1 << 19), "batch": rng.choice([4096, 8192, 16384]),
                "epochs": 1}
    if path == "ensemble":
        return {"path": path, "members": rng.randint(3, 8), "low": 64, "high": rng.randint(96, 256),
                "steps": rng.randint(4, 10), "substeps": rng.randint(3, 6), "dt": 1.0, "tuned": True,
                "draw": rng.randint(0, 1 << 20)}
    kind = rng.choice(["bubble", "cold_pool", "moist", "moist", "mountain", "moist_mountain"])
    nx, ny = _log_int(rng, 32, 700), _log_int(rng, 32, 700)
    if path == "host":
        kind, nx, ny = "moist", min(nx, 400), min(ny, 400)
    nz = rng.randint(24, 80)
    # level spacing near 250 m at dt 1 s (an acoustic limit of the scheme)
    z_top = 250.0 * nz
    case = _leg("", kind, nx, ny, nz, 1 if path == "host" else rng.randint(4, 20), rng.randint(3, 6),
                0.5 if kind in ("bubble", "cold_pool", "mountain") else 1.0,
                1000.0 if kind in ("bubble", "cold_pool", "mountain") else 3000.0, z_top,
                open_sides=rng.random() < 0.4, tuned=rng.random() < 0.5,
                surrogate=kind == "moist" and rng.random() < 0.15)
    case["path"] = path
    del case["name"]
    return case


def _moist(kind):
    return kind.startswith("moist")


def _hilly(kind):
    return kind.endswith("mountain")


def _members(case):
    """The members of an ensemble case as leg cases: uneven sizes, mixed kinds."""
    r = np.random.default_rng(case["draw"])
    out = []
    for m in range(case["members"]):
        kind = ("bubble", "cold_pool", "mountain", "moist")[m % 4]
        nx, ny = (int(v) for v in r.integers(case["low"], case["high"] + 1, 2))
        nz = int(r.choice([40, 64, 80]))
        out.append(_leg("", kind, nx, ny, nz, case["steps"], case["substeps"], case["dt"],
                        3000.0 if kind == "moist" else 1000.0, 250.0 * nz))
    return out


# --------------------------------------------------------------------------------------
# inputs: what the library's case builders give, from the seed alone
def _terrain(case, r):
    """An Agnesi hill, off the centre by the seed."""
    nx, ny = case["nx"], case["ny"]
    cx, cy = (0.5 + 0.1 * (r.random() - 0.5)) * nx, (0.5 + 0.1 * (r.random() - 0.5)) * ny
    a = max(10.0, 0.05 * nx)
    x, y = (np.arange(nx) + 0.5 - cx) / a, (np.arange(ny) + 0.5 - cy) / a
    return (400.0 / (1.0 + x[None, :] ** 2 + y[:, None] ** 2)).astype(np.float32)


def _eta(case):
    """Level interfaces: uniform, or (mountain wave) stretched towards the top."""
    nz = case["nz"]
    s = np.arange(nz + 1) / nz
    return s if case["kind"] != "mountain" else 0.7 * s + 0.3 * s * s


def _weight(eta):
    """Hybrid-height terrain weight with the default taper of 0.25."""
    s = np.clip((eta - 0.25) / 0.75, 0.0, 1.0)
    return np.where(eta <= 0.25, 1.0, 1.0 - s * s * (3.0 - 2.0 * s))


def _heights(case, terrain):
    """Cell-centre and interface heights, FP64 (nz[+1], ny, nx) or (nz[+1], 1, 1)."""
    ei = _eta(case)
    ec = 0.5 * (ei[1:] + ei[:-1])
    h = np.zeros((1, 1)) if terrain is None else terrain.astype(np.float64)
    at = lambda e: e[:, None, None] * case["z_top"] + _weight(e)[:, None, None] * h[None]  # noqa: E731
    return at(ec), at(ei)


def _host(shape, dtype=torch.float32):
    return torch.empty(shape, dtype=dtype, pin_memory=torch.cuda.is_available())


def _state(case, seed):
    """The initial state: host tensors (page-locked) and the terrain of the case."""
    r = np.random.default_rng(seed)
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    kind, nx, ny, nz = case["kind"], case["nx"], case["ny"], case["nz"]
    terrain = _terrain(case, r) if _hilly(kind) else None
    zc, _ = _heights(case, terrain)
    z = torch.tensor(zc, device=dev)
    cp = RD / KAPPA
    # basic state: constant stability (analytic Exner function), 300 K neutral for the bubbles
    n2 = {"mountain": 1.0e-4, "moist": 1.2e-4, "moist_mountain": 1.2e-4}.get(kind, 0.0)
    th0 = 288.0 if kind == "mountain" else 300.0
    if n2:
        theta = th0 * torch.exp(n2 * z / GRAVITY)
        exner = 1.0 - GRAVITY * GRAVITY / (cp * th0 * n2) * (1.0 - torch.exp(-n2 * z / GRAVITY))
    else:
        theta = torch.full_like(z, th0)
        exner = 1.0 - GRAVITY * z / (cp * th0)
    p = P0 * exner.clamp(min=0.05) ** (1.0 / KAPPA)
    rt = (P0 / RD) * (p / P0) ** (1.0 - KAPPA)
    full = (nz, ny, nx)
    theta, rt, p, exner = (t.expand(full).clone() for t in (theta, rt, p, exner))
    x = torch.arange(nx, device=dev, dtype=torch.float64)[None, None, :] + 0.5
    y = torch.arange(ny, device=dev, dtype=torch.float64)[None, :, None] + 0.5
    cx, cy = (0.4 + 0.2 * r.random()) * nx, (0.4 + 0.2 * r.random()) * ny
    rx, ry = max(4.0, 0.15 * nx), max(4.0, 0.15 * ny)

    def blob(zmid, depth):
        d = torch.sqrt(((x - cx) / rx) ** 2 + ((y - cy) / ry) ** 2 + ((z - zmid) / depth) ** 2)
        return torch.where(d < 1.0, torch.cos(0.5 * math.pi * d) ** 2, torch.zeros_like(d))

    if kind == "bubble":
        theta += (1.5 + r.random()) * blob(2000.0, 1500.0)
    elif kind == "cold_pool":
        theta -= (8.0 + 4.0 * r.random()) * blob(0.0, 2500.0)
    theta += 0.1 * torch.randn(full, device=dev, dtype=torch.float64, generator=gen) * (z < 1500.0)
    rho = rt / theta
    wind = {"mountain": 10.0, "moist_mountain": 8.0, "moist": 6.0}.get(kind, 0.0)
    out = {}

    def keep(name, t):
        out[name] = _host(t.shape, torch.float64 if name == "precip" else torch.float32).copy_(t)

    keep("rho", rho)
    keep("rho_theta", rt)
    u = torch.zeros((nz, ny, nx + 1), device=dev, dtype=torch.float64)
    v = torch.zeros((nz, ny + 1, nx), device=dev, dtype=torch.float64)
    u[:, :, :nx] = wind * rho * (1.0 + 0.5 * z / case["z_top"])
    v[:, :ny] = 0.25 * wind * rho
    u[:, :, nx], v[:, ny] = (u[:, :, nx - 1], v[:, ny - 1]) if case["open"] else (u[:, :, 0], v[:, 0])
    keep("u", u)
    keep("v", v)
    keep("w", torch.zeros((nz + 1, ny, nx), device=dev, dtype=torch.float64))
    if _moist(kind):
        # a saturated cloud over a rain shaft in a moist boundary layer
        cloud = blob(2500.0, 1500.0) * (1.0 + 0.2 * torch.rand(full, device=dev, dtype=torch.float64, generator=gen))
        rh = torch.maximum(0.9 * torch.exp(-(z - 2000.0).clamp(min=0.0) / 1500.0), 1.005 * (cloud > 0.0))
        keep("qv", rho * (rh * _qsat(theta * exner, p)).clamp(min=1.0e-5))
        keep("qc", rho * (8.0e-4 * cloud))
        keep("qr", rho * (4.0e-4 * torch.maximum(cloud, blob(800.0, 1500.0))))
        keep("precip", torch.zeros((ny, nx), device=dev, dtype=torch.float64))
    return out, terrain


def _damping(case, state):
    """The mountain wave's Rayleigh layer: bottom, rate and the wind it relaxes to."""
    mean = lambda k: state[k].numpy().mean(axis=(1, 2), dtype=np.float64)  # noqa: E731
    return 0.7 * case["z_top"], 0.05, mean("u"), mean("v")


def _arrays(state):
    return {k: t.numpy() for k, t in state.items()}


def _spec(gwm, case, terrain):
    grid = gwm.GridSpec(case["nx"], case["ny"], case["nz"], dx=case["spacing"], dy=case["spacing"],
                        z_top=case["z_top"], periodic_x=not case["open"], periodic_y=not case["open"], terrain=terrain,
                        eta_interfaces=_eta(case) if case["kind"] == "mountain" else None)
    member = gwm.MemberSpec(step=gwm.StepConfig(dt=case["dt"], fast_substeps=case["substeps"]),
                            rain=gwm.WarmRainConfig(dt=case["dt"], rain_terminal_velocity=FALL_SPEED),
                            moist=_moist(case["kind"]))
    return grid, member


def _scalar_inputs(case, seed):
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    q = torch.rand((case["nz"], case["ny"], case["nx"]), device=dev, generator=gen)
    return q, dict(u_adv=20.0, v_adv=10.0, dt=10.0, dx=1000.0, dy=1000.0)


def _train_inputs(case, seed):
    """Samples of the ranges the warm-rain recorder writes, with smooth targets."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    a = torch.rand((case["samples"], 7), device=dev, generator=gen)
    low = torch.tensor([240.0, 3.0e4, 0.4, 1.0e-5, 0.0, 0.0, 1.0], device=dev)
    high = torch.tensor([305.0, 1.0e5, 1.2, 0.02, 2.0e-3, 1.0e-3, 1.0], device=dev)
    x = (low + (high - low) * a).contiguous()
    y = torch.stack([torch.tanh(2.0 * a[:, 3] - a[:, 0]), 1.0e-3 * a[:, 4], 5.0e-3 * (1.0 - a[:, 3]) * a[:, 5],
                     2.0 * (a[:, 3] - a[:, 0]) * a[:, 1], -8.0e-4 * (a[:, 3] - a[:, 0])], dim=1).contiguous()
    return x, y


def prepare(case, seed):
    gwm = _gwm()
    path = case["path"]
    if path == "scalar":
        q0, opts = _scalar_inputs(case, seed)
        return {"case": case, "q0": q0, "q": torch.empty_like(q0), "opts": opts}
    if path == "train":
        x, y = _train_inputs(case, seed)
        return {"case": case, "x": x, "y": y}
    members = _members(case) if path == "ensemble" else [case]
    grids, specs, inputs, damping = [], [], [], []
    for i, c in enumerate(members):
        state, terrain = _state(c, seed + 1000 * i)
        grid, member = _spec(gwm, c, terrain)
        grids.append(grid)
        specs.append(member)
        inputs.append(state)
        damping.append(_damping(c, state) if c["kind"] == "mountain" else None)
    model = gwm.Model(grids, specs)
    for i, d in enumerate(damping):
        if d is not None:
            model.set_damping(d[0], d[1], u_ref=d[2], v_ref=d[3], member=i)
    if case.get("surrogate"):
        w = np.load(os.path.join(list(gwm.__path__)[0], "surrogate_c3.npz"))
        model.set_rain_surrogate(w["params"], w["norm"], w["range"])
    arrays = [_arrays(s) for s in inputs]
    if case["tuned"]:
        for i, a in enumerate(arrays):
            model.upload(a, member=i)
        model.autotune(whole_step=path == "ensemble")
    if path != "host":
        model.use_graph(True)
    results = [{k: _host(t.shape, t.dtype) for k, t in s.items()} for s in inputs]
    return {"case": case, "model": model, "in": arrays, "out": [_arrays(r) for r in results],
            "keep": (inputs, results)}


def run(state):
    gwm = _gwm()
    case = state["case"]
    path = case["path"]
    if path == "scalar":
        state["q"].copy_(state["q0"])
        gwm.scalar_ssprk3(state["q"], nsteps=case["steps"], periodic_x=not case["open"],
                          periodic_y=not case["open"], **state["opts"])
        return state["q"]
    if path == "train":
        params, norm, rng, loss = gwm.mlp_train(state["x"], state["y"], case["samples"], epochs=case["epochs"],
                                                batch=case["batch"], seed=3)
        return [params, norm, rng, loss]
    model = state["model"]
    if path == "host":
        return model.step_host(state["in"][0], state["out"][0])
    for i, a in enumerate(state["in"]):
        model.upload(a, member=i)
    model.step(case["steps"])
    for i, a in enumerate(state["out"]):
        model.download(member=i, out=a)
    return state["out"] if path == "ensemble" else state["out"][0]


# --------------------------------------------------------------------------------------
# bytes and operations a pass cannot do without
def _leg_work(case):
    cells = case["nx"] * case["ny"] * case["nz"]
    moist = _moist(case["kind"])
    nf = 8 if moist else 5
    hilly = _hilly(case["kind"])
    # FP32 fields read and written once by each operator: slow stages 5 (+3 increments, +5
    # blend partner) in and 5 out; an acoustic substep 6 in (2 the first of a stage, 9 the
    # last of the step) and 4 out, terrain heights in; tracers rho, 3 momenta, 3 (+3) in and
    # 3 out; rain 5 in, 4 out
    fields = (10 + 2 * 18) + 3 * (case["substeps"] * (10 + hilly) - 3)
    flops = 3 * 240 + 3 * case["substeps"] * (45 + (60 if hilly else 0))
    if moist:
        fields += (7 + 3) + 2 * (10 + 3) + 9
        flops += 3 * 90 + 120
        if case["surrogate"]:  # the network on a tenth of the cells
            flops += 0.1 * 2 * (7 * 64 + 2 * 64 * 64 + 64 * 5)
    return 4.0 * cells * (case["steps"] * fields + 2 * nf), float(cells) * case["steps"] * flops


def work(case):
    path = case["path"]
    if path == "scalar":
        cells = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 4.0 * cells * (2 + case["steps"] * 8), "flops": 30.0 * cells * case["steps"]}
    if path == "train":
        w = 7 * 64 + 2 * 64 * 64 + 64 * 5
        return {"bytes": 48.0 * case["samples"] * case["epochs"], "flops": 6.0 * w * case["samples"] * case["epochs"]}
    parts = [_leg_work(c) for c in (_members(case) if path == "ensemble" else [case])]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


# --------------------------------------------------------------------------------------
# the step in 64 bits
def _qsat(t, p):
    tc = t - float(np.float32(273.15))
    es = 100.0 * float(np.float32(6.112)) * torch.exp(float(np.float32(17.67)) * tc / (tc + 243.5).clamp(min=1.0e-6))
    eps = RD / RV
    return (eps * es / (p - (1.0 - eps) * es).clamp(min=1000.0)).clamp(min=0.0, max=float(np.float32(0.05)))


def _eos(rho, rt):
    return P0 * (rho * RD * (rt / rho.clamp(min=1.0e-6)) / P0).clamp(min=1.0e-6) ** (1.0 / (1.0 - KAPPA))


def _eos_rho(p, theta):
    return p / (RD * theta * (p / P0).clamp(min=1.0e-6) ** KAPPA).clamp(min=1.0e-6)


def _upwind(a, low, high):
    return a * torch.where(a >= 0, low, high)


def _swap(t):
    return None if t is None else t.transpose(-1, -2)


class _Exact:
    """One member in 64 bits: fields (z, y, x), faces with both end faces of their axis."""

    def __init__(self, case, state, terrain, damping, device):
        f64 = lambda a: torch.as_tensor(a, dtype=torch.float64, device=device)  # noqa: E731
        self.case, self.dt, self.open = case, case["dt"], case["open"]
        self.d = float(case["spacing"])
        self.s = {k: f64(t) for k, t in state.items()}
        self.nz = case["nz"]
        self.hilly = terrain is not None and bool((np.abs(terrain) > 1.0e-6).any())
        zc, zi = _heights(case, terrain)
        zf = np.zeros_like(zi)
        zf[1:-1] = 1.0 / np.maximum(zc[1:] - zc[:-1], 1.0e-6)
        full = lambda a: f64(a).expand(a.shape[0], case["ny"], case["nx"])  # noqa: E731
        self.idc, self.idf = full(1.0 / np.maximum(zi[1:] - zi[:-1], 1.0e-6)), full(zf)
        self.zc = self.pad_metric(full(zc))
        self.idc_pad = self.pad_metric(self.idc)
        self.damp = None
        if damping is not None:
            bottom, rate, u_ref, v_ref = damping
            eta = _eta(case)

            def tau(z):
                a = np.sin(0.5 * np.pi * np.clip((z - bottom) / (case["z_top"] - bottom), 0.0, 1.0))
                return f64(rate * a * a)[:, None, None]

            self.damp = (tau(0.5 * (eta[1:] + eta[:-1]) * case["z_top"]), tau(eta * case["z_top"])[1:-1],
                         f64(u_ref)[:, None, None], f64(v_ref)[:, None, None])

    # halo of one cell: the periodic image, or zero beyond an open side
    def _pad(self, t, dim, low, high):
        a, b = t.narrow(dim, low, 1), t.narrow(dim, high, 1)
        if self.open:
            a, b = torch.zeros_like(a), torch.zeros_like(b)
        return torch.cat([a, t, b], dim)

    def pad(self, t, fx=0, fy=0):
        """fx, fy: the axis holds faces (both ends), so the image skips the shared face."""
        t = self._pad(t, 2, t.shape[2] - 1 - fx, fx)
        return self._pad(t, 1, t.shape[1] - 1 - fy, fy)

    def pad_metric(self, t):
        keep, self.open = self.open, False
        t = self.pad(t)
        self.open = keep
        return t

    def dpdz(self, p):
        if self.nz == 1:
            return torch.zeros_like(p)
        z, out = self.zc, torch.empty_like(p)
        out[1:-1] = (p[2:] - p[:-2]) / (z[2:] - z[:-2]).clamp(min=1.0e-6)
        out[0] = (p[1] - p[0]) / (z[1] - z[0]).clamp(min=1.0e-6)
        out[-1] = (p[-1] - p[-2]) / (z[-1] - z[-2]).clamp(min=1.0e-6)
        return out

    def gradient(self, p, dpdz, z):
        """Pressure gradient at the X faces (0 .. nx) of owned rows; inputs padded."""
        p, dpdz, z = p[:, 1:-1], dpdz[:, 1:-1], z[:, 1:-1]
        slope = (z[..., 1:] - z[..., :-1]) / self.d
        return (p[..., 1:] - p[..., :-1]) / self.d - slope * 0.5 * (dpdz[..., 1:] + dpdz[..., :-1])

    def closed(self, t):
        """Face tendency with the faces of open sides left alone."""
        if self.open:
            t[..., 0] = 0.0
            t[..., -1] = 0.0
        return t

    def face_tendency(self, q, uc, vc, wc, idc, p, dpdz, z):
        """Tendency of the X-face momentum; the Y faces are the transposed call."""
        c = q[:, 1:-1, 1:-1]
        flw = _upwind(uc[:, 1:-1, :-1], q[:, 1:-1, :-2], c)
        fle = _upwind(uc[:, 1:-1, 1:], c, q[:, 1:-1, 2:])
        va = 0.5 * (vc[..., :-1] + vc[..., 1:])
        fls = _upwind(va[:, :-2], q[:, :-2, 1:-1], c)
        fln = _upwind(va[:, 1:-1], c, q[:, 2:, 1:-1])
        if self.open:
            fls[:, 0] = 0.0
            fln[:, -1] = 0.0
        wa = 0.5 * (wc[:, 1:-1, :-1] + wc[:, 1:-1, 1:])
        fz = torch.zeros((self.nz + 1,) + tuple(c.shape[1:]), dtype=c.dtype, device=c.device)
        fz[1:-1] = _upwind(wa[:-1], c[:-1], c[1:])
        idz = 0.5 * (idc[:, 1:-1, :-1] + idc[:, 1:-1, 1:])
        t = -((fle - flw) / self.d + (fln - fls) / self.d + (fz[1:] - fz[:-1]) * idz)
        return t - self.gradient(p, dpdz, z)

    def flux_divergence(self, q, u, v, w):
        """Upwind flux divergence of a padded cell field carried by the mass fluxes."""
        c = q[:, 1:-1, 1:-1]
        fx = _upwind(u, q[:, 1:-1, :-1], q[:, 1:-1, 1:])
        fy = _upwind(v, q[:, :-1, 1:-1], q[:, 1:, 1:-1])
        fz = _upwind(w, torch.cat([c[:1], c]), torch.cat([c, c[-1:]]))
        return self.divergence(fx, fy, fz)

    def divergence(self, fx, fy, fz):
        return (fx[..., 1:] - fx[..., :-1]) / self.d + (fy[:, 1:] - fy[:, :-1]) / self.d + (fz[1:] - fz[:-1]) * self.idc

    def slow(self, rho, rt, u, v, w):
        r, t = self.pad(rho), self.pad(rt)
        th, p = t / r.clamp(min=1.0e-6), _eos(r, t)
        up, vp, wp = self.pad(u, fx=1), self.pad(v, fy=1), self.pad(w)
        rr = r.clamp(min=1.0e-6)
        uc = 0.5 * (up[..., :-1] + up[..., 1:]) / rr
        vc = 0.5 * (vp[:, :-1] + vp[:, 1:]) / rr
        wc = 0.5 * (wp[:-1] + wp[1:]) / rr
        t_rho = -self.divergence(u, v, w)
        t_rt = -self.flux_divergence(th, u, v, w)
        g = self.dpdz(p)
        t_u = self.face_tendency(up, uc, vc, wc, self.idc_pad, p, g, self.zc)
        t_v = _swap(self.face_tendency(_swap(vp), _swap(vc), _swap(uc), _swap(wc), _swap(self.idc_pad), _swap(p),
                                       _swap(g), _swap(self.zc)))
        c = wp[1:-1, 1:-1, 1:-1]
        ua, va = 0.5 * (uc[:-1] + uc[1:]), 0.5 * (vc[:-1] + vc[1:])
        flw = _upwind(ua[:, 1:-1, :-2], wp[1:-1, 1:-1, :-2], c)
        fle = _upwind(ua[:, 1:-1, 1:-1], c, wp[1:-1, 1:-1, 2:])
        fls = _upwind(va[:, :-2, 1:-1], wp[1:-1, :-2, 1:-1], c)
        fln = _upwind(va[:, 1:-1, 1:-1], c, wp[1:-1, 2:, 1:-1])
        if self.open:
            flw[..., 0], fle[..., -1], fls[:, 0], fln[:, -1] = 0.0, 0.0, 0.0, 0.0
        fz = _upwind(wc[:, 1:-1, 1:-1], w[:-1], w[1:])
        t_w = torch.zeros_like(w)
        t_w[1:-1] = -((fle - flw) / self.d + (fln - fls) / self.d + (fz[1:] - fz[:-1]) * self.idf[1:-1])
        tc = th[:, 1:-1, 1:-1]
        ref = tc.mean(dim=(1, 2), keepdim=True)
        tf, trf = 0.5 * (tc[1:] + tc[:-1]), 0.5 * (ref[1:] + ref[:-1])
        t_w[1:-1] += 0.5 * (rho[1:] + rho[:-1]) * GRAVITY * (tf - trf) / trf.clamp(min=1.0e-6)
        if self.damp is not None:
            tau_c, tau_f, u_ref, v_ref = self.damp
            t_u -= tau_c * (u - u_ref)
            t_v -= tau_c * (v - v_ref)
            t_w[1:-1] -= tau_f * w[1:-1]
        return t_rho, t_rt, self.closed(t_u), _swap(self.closed(_swap(t_v))), t_w

    def column_reference(self, rho, th, p):
        z, pref, rref = self.zc[:, 1:-1, 1:-1], torch.empty_like(rho), torch.empty_like(rho)
        pref[0] = p[0]
        rref[0] = _eos_rho(pref[0], th[0])
        for k in range(1, self.nz):
            dz = z[k] - z[k - 1]
            pn = (pref[k - 1] - GRAVITY * rref[k - 1] * dz).clamp(min=1.0)
            for _ in range(4):
                pn = (pref[k - 1] - GRAVITY * 0.5 * (rref[k - 1] + _eos_rho(pn, th[k])) * dz).clamp(min=1.0)
            pref[k], rref[k] = pn, _eos_rho(pn, th[k])
        return rref, pref

    def fast(self, rho, rt, u, v, w):
        n = max(1, self.case["substeps"])
        dtf = self.dt / n
        th = self.pad(rt) / self.pad(rho).clamp(min=1.0e-6)
        tc = th[:, 1:-1, 1:-1]
        u0, v0, w0 = u, v, w
        for _ in range(n):
            r = self.pad(rho)
            p = _eos(r, r * th)
            pc = p[:, 1:-1, 1:-1]
            if self.hilly:
                rref, pref = self.column_reference(rho, tc, pc)
            else:
                rref, pref = rho.mean(dim=(1, 2), keepdim=True), pc.mean(dim=(1, 2), keepdim=True)
            g = self.dpdz(p)
            u = u - dtf * self.closed(self.gradient(p, g, self.zc))
            v = v - dtf * _swap(self.closed(self.gradient(_swap(p), _swap(g), _swap(self.zc))))
            pp, rp = pc - pref, rho - rref
            w = w.clone()
            w[1:-1] += dtf * (-(pp[1:] - pp[:-1]) * self.idf[1:-1] - GRAVITY * 0.5 * (rp[1:] + rp[:-1]))
            rho = (rho - dtf * self.divergence(u - u0, v - v0, w - w0)).clamp(min=1.0e-6)
        return rho, rho * tc, u, v, w

    def step(self):
        q0 = tuple(self.s[k] for k in STATE)
        q = q0
        for a, b in ((0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)):
            new = [x + self.dt * t for x, t in zip(q, self.slow(*q))]
            new[0], new[1] = new[0].clamp(min=1.0e-6), new[1].clamp(min=1.0e-6)
            q = self.fast(*(a * x + b * y for x, y in zip(q0, new)))
        self.s.update(zip(STATE, q))
        if _moist(self.case["kind"]):
            self.tracers()
            self.rain()

    def tracers(self):
        rho, u, v, w = (self.s[k] for k in ("rho", "u", "v", "w"))
        r = self.pad(rho).clamp(min=1.0e-6)
        for name in TRACERS:
            q0 = q = self.s[name]
            for a, b in ((0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)):
                new = (q - self.dt * self.flux_divergence(self.pad(q) / r, u, v, w)).clamp(min=0.0)
                q = a * q0 + b * new
            self.s[name] = q

    def rain(self):
        threshold, rate, evaporation = (float(np.float32(x)) for x in (1.0e-4, 1.0e-3, 5.0e-3))
        rho, rt = self.s["rho"].clamp(min=1.0e-6), self.s["rho_theta"]
        th, p = rt / rho, _eos(rho, rt)
        exner = (p / P0).clamp(min=1.0e-6) ** KAPPA
        heat = LV / (RD / KAPPA * exner)
        qv, qc, qr = ((self.s[k] / rho).clamp(min=0.0) for k in TRACERS)
        qs = _qsat(th * exner, p)
        change = torch.where(qv > qs, torch.minimum(qv - qs, qv), -torch.minimum(qs - qv, qc))
        qv, qc, th = qv - change, qc + change, th + heat * change
        excess = (qc - threshold).clamp(min=0.0)
        conversion = torch.minimum(excess, self.dt * rate * excess)
        qc, qr = qc - conversion, qr + conversion
        p = _eos(rho, rho * th)
        qs = _qsat(th * (p / P0).clamp(min=1.0e-6) ** KAPPA, p)
        ev = torch.minimum(qr, self.dt * evaporation * torch.minimum((qs - qv).clamp(min=0.0), qr))
        qr, qv, th = qr - ev, qv + ev, th - heat * ev
        fall = (FALL_SPEED * self.dt * self.idc).clamp(min=0.0, max=1.0) * (rho * qr) / self.idc
        above = torch.cat([fall[1:], torch.zeros_like(fall[:1])])
        self.s.update(rho_theta=rho * th, qv=rho * qv, qc=rho * qc, qr=rho * qr + (above - fall) * self.idc,
                      precip=self.s["precip"] + fall[0])


def _exact_leg(case, seed):
    device = _device()
    state, terrain = _state(case, seed)
    damping = _damping(case, state) if case["kind"] == "mountain" else None
    e = _Exact(case, state, terrain, damping, device)
    del state
    for _ in range(case["steps"]):
        e.step()
    return {k: t.cpu() for k, t in e.s.items()}


def _exact_scalar(case, seed):
    q, o = _scalar_inputs(case, seed)
    q = q.double()

    def stage(q):
        x, y = torch.roll(q, 1, 2), torch.roll(q, 1, 1)
        if case["open"]:
            x[:, :, 0] = 0.0
            y[:, 0] = 0.0
        return q - o["dt"] * (o["u_adv"] * (q - x) / o["dx"] + o["v_adv"] * (q - y) / o["dy"])

    for _ in range(case["steps"]):
        q1 = stage(q)
        q2 = 0.75 * q + 0.25 * stage(q1)
        q = q / 3.0 + 2.0 / 3.0 * stage(q2)
    return q


def exact(case, seed):
    """What run() returns, in 64 bits.  None for the largest grids (over 20 s), for the
    learned warm rain (BF16 inference with its own fallback rules) and for the training
    (its shuffle and initial weights are the library's)."""
    path = case["path"]
    if path == "scalar":
        return _exact_scalar(case, seed)
    if path == "train" or case.get("surrogate"):
        return None
    if path == "ensemble":
        return [_exact_leg(c, seed + 1000 * i) for i, c in enumerate(_members(case))]
    if case["nx"] * case["ny"] * case["nz"] * case["steps"] * case["substeps"] > EXACT_MOST:
        return None
    return _exact_leg(case, seed)
