"""Performance cases: the work users of this framework have it do, through its
public entry points, with the 64-bit values each case has to produce.

A case is a dict of plain values.  `kind` says which entry point it goes
through:

  march     a device-resident grid (`Grid`): a stored state put in, `steps`
            main-loop iterations, the new state copied out on the device
  ensemble  many independent blast grids of uneven sizes (`Batch`): generated
            on the GPU, `steps` iterations, every state downloaded
  dropin    the reference's own entry points on a host Grid (`DropInLoop`)
  gradient  dJ/d(initial state) of `steps` iterations (`Grid.adjoint_gradient`)
  tangent   the tangent-linear model of `steps` iterations (`Grid.tlm`)

Every pass is a short run from the same initial state, as in a parameter
study; the simulation clock of a march goes on from pass to pass.

`exact` marches the same initial state with a plain torch restatement of the
CTU + constrained-transport scheme (characteristic PLM, Roe with the HLLE
fallback or HLLE), and differentiates it with torch's autograd.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import athena_cuda_b200 as ab
from athena_cuda_b200 import dropin

NG = ab.NGHOST
GAMMA = 1.6666666666666667
COUR = 0.8
TLIM = 1.0e6          # never reached: a pass is bounded by its steps
PERIODIC = "4444"     # boundary flags ix1 ox1 ix2 ox2: 1 reflecting, 2 outflow, 4 periodic
ENSEMBLE_SIZES = (64, 96, 128, 192, 256, 384, 512)
EXACT_STATE_SECONDS = 0.05   # about what one iteration of the torch restatement takes

# FP64 additions, multiplications, divisions and square roots of one
# zone-cycle (the counting build of the CPU oracle, field loop, Roe), and the
# planes a step reads and writes once.
FLOPS_PER_ZONE = 4970.0
STATE_BYTES = 8 * ab.NPLANES


def listed():
    return [
        # the smallest configured wave: a step is launches and dependent latency
        _march("wave_32x16", "wave", 32, 16, 32),
        # the example input of the wave problem's size class, with the HLLE option
        _march("wave_128x64_hlle", "wave", 128, 64, 40, flux="hlle"),
        # the reference's standard blast (examples/athinput.blast)
        _march("blast_200x300", "blast", 200, 300, 20),
        # an odd-sized box with walls and outflow, as the parity tests use
        _march("blast_333x217_walls", "blast", 333, 217, 20, bc="1221"),
        # the field loop's example size
        _march("loop_1024x512", "loop", 1024, 512, 10),
        # the largest configured grid, the headline benchmark
        _march("loop_2048x2048", "loop", 2048, 2048, 5),
        # a slice of the batched blast ensemble: uneven sizes, own dt each
        {"name": "ensemble_24", "kind": "ensemble", "n": 24, "steps": 48, "flux": "roe"},
        # a program of the reference relinked: host Grid, copies in every call
        {"name": "dropin_200x300", "kind": "dropin", "problem": "blast", "nx1": 200, "nx2": 300, "steps": 8,
         "flux": "roe", "bc": PERIODIC},
        # a small gradient, as a test or a first experiment asks for
        _sens("gradient_64x48", "gradient", 64, 48, 10),
        # the configured gradient's grid, every step's tape kept in memory
        _sens("gradient_256x256", "gradient", 256, 256, 40),
        # a gradient whose checkpoints do not fit: snapshots and recomputation
        _sens("gradient_512x384_snapshots", "gradient", 512, 384, 24, snapshots=6),
        # one directional derivative
        _sens("tangent_128x128", "tangent", 128, 128, 10),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    flux = "hlle" if rng.random() < 0.2 else "roe"
    kind = rng.choice(["march"] * 6 + ["gradient"] * 2 + ["ensemble", "dropin", "tangent"])
    if kind == "march":
        problem = rng.choice(["wave", "blast", "blast", "loop", "loop"])
        nx1, nx2 = log_int(16, 1700), log_int(16, 1700)
        bc = PERIODIC
        if problem == "blast" and rng.random() < 0.5:   # periodic needs both sides of a direction
            bc = "".join(rng.choice(["44", "11", "22", "12", "21"]) for _ in range(2))
        c = _march("", problem, nx1, nx2, rng.randint(16, 40) if nx1 * nx2 < 1.0e5 else 8, flux=flux,
                   bc=bc)
    elif kind == "ensemble":
        c = {"kind": "ensemble", "n": rng.randint(6, 24), "steps": rng.randint(24, 48), "flux": flux}
    elif kind == "dropin":
        c = {"kind": "dropin", "problem": rng.choice(["blast", "loop"]), "nx1": log_int(24, 500),
             "nx2": log_int(24, 500), "steps": rng.randint(4, 8), "flux": flux, "bc": PERIODIC}
    else:
        nx1, nx2 = log_int(24, 300), log_int(24, 300)
        c = _sens("", kind, nx1, nx2, rng.randint(5, 20), flux=flux,
                  snapshots=rng.choice([0, 4]) if kind == "gradient" else 0)
    c.pop("name", None)
    return c


def _march(name, problem, nx1, nx2, steps, flux="roe", bc=PERIODIC):
    return {"name": name, "kind": "march", "problem": problem, "nx1": nx1, "nx2": nx2, "steps": steps,
            "flux": flux, "bc": bc}


def _sens(name, kind, nx1, nx2, steps, flux="roe", snapshots=0):
    return {"name": name, "kind": kind, "problem": "loop", "nx1": nx1, "nx2": nx2, "steps": steps,
            "flux": flux, "bc": PERIODIC, "snapshots": snapshots}


# ---------------------------------------------------------------------------
# what a program has before the call
# ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "ensemble":
        items = _instances(case)
        batch = ab.Batch([_config(c) for c in items])
        params = [ab.Params.from_blocks({"problem": _blast(c, seed)}) for c in items]
        return {"case": case, "batch": batch, "params": params}
    planes = _initial(case, seed)
    cfg = _config(case)
    if case["kind"] == "dropin":
        host = dropin.HostGrid(planes.cpu().numpy(), (cfg.x1max - cfg.x1min) / cfg.nx1,
                               (cfg.x2max - cfg.x2min) / cfg.nx2, cfg.x1min, cfg.x2min)
        loop = dropin.DropInLoop(host, GAMMA, COUR, _bc(case), cfg.flux)
        return {"case": case, "loop": loop, "host": host, "dt": host.grid.dt,
                "start": [a.copy() for a in (host.U, *host.B)]}
    grid = ab.Grid.create(cfg)
    grid.upload(planes.cpu().numpy())
    grid.set_bvals()
    grid.new_dt()
    state = {"case": case, "grid": grid}
    if case["kind"] == "march":
        state["start"] = torch.empty(planes.shape, dtype=torch.float64, device="cuda")
        state["out"] = torch.empty_like(state["start"])
        _copy(grid, "athb_rect_pack", state["start"])
        grid.synchronize()
    elif case["kind"] == "gradient":
        grid.keep_adjoint_workspace()   # as an optimiser that calls it again does
        state["budget"] = case["snapshots"] * _plane_doubles(case) * STATE_BYTES
    else:
        state["direction"] = _direction(case, seed).cpu().numpy()
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "march":
        grid = state["grid"]
        _copy(grid, "athb_rect_unpack", state["start"])
        grid.new_dt()
        grid.run(case["steps"])
        _copy(grid, "athb_rect_pack", state["out"])
        s = grid.status()
        return {"state": state["out"], "dt": s["dt"], "time": s["time"]}
    if case["kind"] == "ensemble":
        batch = state["batch"]
        for k, p in enumerate(state["params"]):
            batch.generate(k, "blast", p)
        batch.prepare()
        batch.run(case["steps"])
        got = [batch.download(k) for k in range(batch.n)]
        return {"states": [g[0] for g in got], "dt": np.array([g[1] for g in got]),
                "time": np.array([g[2] for g in got])}
    if case["kind"] == "dropin":
        host = state["host"]
        for a, b in zip((host.U, *host.B), state["start"]):
            a[...] = b
        host.grid.dt, host.grid.time, host.grid.nstep = state["dt"], 0.0, 0
        state["loop"].steps(case["steps"])
        return {"state": host.planes(), "dt": float(host.grid.dt), "time": float(host.grid.time)}
    if case["kind"] == "gradient":
        J, g, _ = state["grid"].adjoint_gradient(case["steps"], state["budget"])
        return {"J": J, "gradient": g}
    J, dJ, ds = state["grid"].tlm(case["steps"], state["direction"], want_state=True)
    return {"J": J, "dJ": dJ, "dS": ds}


def _copy(grid, entry, tensor):
    """The whole state between the grid and a tensor on the GPU."""
    ab._check(getattr(ab.lib(), entry)(grid._h, C.c_int(0), C.c_int(grid.sx), C.c_int(0), C.c_int(grid.sy),
                                       C.c_void_p(tensor.data_ptr())))


def work(case):
    if case["kind"] == "ensemble":
        # the mean size of the ensemble's instances
        zones = case["n"] * (sum(ENSEMBLE_SIZES) / len(ENSEMBLE_SIZES)) ** 2
    else:
        zones = case["nx1"] * case["nx2"]
    # forward work alone for march and drop-in; a gradient cannot do without
    # the forward step and about twice its operations backwards, a tangent
    # carries value and derivative
    factor = {"gradient": 3.0, "tangent": 2.0}.get(case["kind"], 1.0)
    return {"bytes": 2.0 * STATE_BYTES * zones, "flops": factor * FLOPS_PER_ZONE * zones * case["steps"]}


def _bc(case):
    return tuple(int(b) for b in case["bc"])


def _box(case):
    """x1min, x1max, x2min, x2max of the case's problem."""
    if case["problem"] == "wave":
        return 0.0, 1.0, 0.0, 0.5
    if case["problem"] == "loop":
        return -1.0, 1.0, -0.5, 0.5
    half = 0.5 * case["nx2"] / case["nx1"]
    return -0.5, 0.5, -half, half


def _config(case):
    x1min, x1max, x2min, x2max = _box(case)
    ix1, ox1, ix2, ox2 = _bc(case)
    return ab.Config(nx1=case["nx1"], nx2=case["nx2"], x1min=x1min, x1max=x1max, x2min=x2min, x2max=x2max,
                     bc_ix1=ix1, bc_ox1=ox1, bc_ix2=ix2, bc_ox2=ox2, gamma=GAMMA, cour_no=COUR, tlim=TLIM,
                     nlim=-1, flux=ab.FLUX_HLLE if case["flux"] == "hlle" else ab.FLUX_ROE, device=0)


def _plane_doubles(case):
    """Doubles of one plane as the framework lays it out (rows of 16)."""
    return ((case["nx1"] + 2 * NG + 15) // 16 * 16) * (case["nx2"] + 2 * NG)


def _instances(case):
    """The ensemble's grids: sides drawn from the configured sizes, fixed for
    a case; the physics of each comes from the seed (`_blast`)."""
    rng = np.random.default_rng(case["n"])
    return [{"kind": "march", "problem": "blast", "nx1": int(rng.choice(ENSEMBLE_SIZES)),
             "nx2": int(rng.choice(ENSEMBLE_SIZES)), "flux": case["flux"], "bc": PERIODIC, "member": k}
            for k in range(case["n"])]


def _blast(case, seed):
    """The problem block of one blast, over the ensemble's ranges."""
    rng = np.random.default_rng([seed, case.get("member", 0)])
    return {"pamb": 0.1, "prat": math.exp(rng.uniform(math.log(10.0), math.log(1000.0))),
            "radius": rng.uniform(0.05, 0.15), "b0": rng.uniform(0.1, 2.0), "angle": rng.uniform(0.0, 180.0)}


# ---------------------------------------------------------------------------
# initial states, made from the seed alone: (11, Nx2+8, Nx1+8), ghosts zero
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _initial(case, seed):
    rng = np.random.default_rng([seed, case.get("member", 0)])
    nx1, nx2 = case["nx1"], case["nx2"]
    x1min, x1max, x2min, x2max = _box(case)
    dx1, dx2 = (x1max - x1min) / nx1, (x2max - x2min) / nx2
    opts = {"dtype": torch.float64, "device": _device()}
    S = torch.zeros((ab.NPLANES, nx2 + 2 * NG, nx1 + 2 * NG), **opts)
    inner = S[:, NG:NG + nx2, NG:NG + nx1]
    # corner coordinates, one beyond the last cell, and the cell centres
    X = (x1min + dx1 * torch.arange(nx1 + 1, **opts))[None, :]
    Y = (x2min + dx2 * torch.arange(nx2 + 1, **opts))[:, None]
    x, y = X[:, :-1] + 0.5 * dx1, Y[:-1] + 0.5 * dx2
    one = torch.ones((nx2, nx1), **opts)
    if case["problem"] == "blast":
        q = _blast(case, seed)
        theta = math.radians(q["angle"])
        rho, v1, v2, v3 = one, 0.0 * one, 0.0 * one, 0.0 * one
        p = torch.where(torch.sqrt(x * x + y * y) < q["radius"], q["pamb"] * q["prat"], q["pamb"]) * one
        b1, b2, b3 = q["b0"] * math.cos(theta), q["b0"] * math.sin(theta), 0.0 * one
        B1f = torch.full((nx2, nx1 + 1), b1, **opts)
        B2f = torch.full((nx2 + 1, nx1), b2, **opts)
    elif case["problem"] == "loop":
        rad, amp = rng.uniform(0.2, 0.35), 1.0e-3 * rng.uniform(0.5, 2.0)
        rho = 1.0 + 0.01 * _smooth_noise(rng, nx1, nx2)
        v1, v2, v3, p, b3 = 2.0 * one, one, 0.0 * one, one, 0.0 * one
        A = amp * torch.clamp(rad - torch.sqrt(X * X + Y * Y), min=0.0)
        B1f, B2f = (A[1:] - A[:-1]) / dx2, -(A[:, 1:] - A[:, :-1]) / dx1
    else:
        # circularly polarised wave, wavevector 2 pi (1, 2), along (1, 2)/sqrt(5)
        k, c, s = 2.0 * math.pi * math.sqrt(5.0), 1.0 / math.sqrt(5.0), 2.0 / math.sqrt(5.0)
        bp, pres, phase = rng.uniform(0.05, 0.2), rng.uniform(0.05, 0.2), rng.uniform(0.0, 2.0 * math.pi)
        A = Y * c - X * s + (bp / k) * torch.cos(k * (X * c + Y * s) + phase)
        B1f, B2f = (A[1:] - A[:-1]) / dx2, -(A[:, 1:] - A[:, :-1]) / dx1
        arg = k * (x * c + y * s) + phase
        rho, p = one, pres * one
        vt = -bp * torch.sin(arg)
        v1, v2, v3 = -vt * s, vt * c, -bp * torch.cos(arg)
        b3 = bp * torch.cos(arg)
    S[8, NG:NG + nx2, NG:NG + nx1 + 1] = B1f
    S[9, NG:NG + nx2 + 1, NG:NG + nx1] = B2f
    inner[5], inner[6] = 0.5 * (B1f[:, 1:] + B1f[:, :-1]), 0.5 * (B2f[1:] + B2f[:-1])
    inner[7], inner[10] = b3, b3
    inner[0], inner[1], inner[2], inner[3] = rho, rho * v1, rho * v2, rho * v3
    inner[4] = (p / (GAMMA - 1.0) + 0.5 * rho * (v1 * v1 + v2 * v2 + v3 * v3)
                + 0.5 * (inner[5] ** 2 + inner[6] ** 2 + inner[7] ** 2))
    return S


def _smooth_noise(rng, nx1, nx2, width=4.0):
    """White noise under a periodic Gaussian of `width` cells, of unit
    standard deviation."""
    noise = torch.as_tensor(rng.standard_normal((nx2, nx1)), device=_device())
    ky = torch.fft.fftfreq(nx2, dtype=torch.float64, device=noise.device)[:, None]
    kx = torch.fft.fftfreq(nx1, dtype=torch.float64, device=noise.device)[None, :]
    kernel = torch.exp(-2.0 * (math.pi * width) ** 2 * (kx * kx + ky * ky))
    s = torch.real(torch.fft.ifft2(torch.fft.fft2(noise) * kernel))
    return s / torch.std(s)


def _direction(case, seed):
    """A smooth density direction at fixed velocity and pressure."""
    rng = np.random.default_rng([seed, 1])
    drho = _smooth_noise(rng, case["nx1"], case["nx2"])
    D = torch.zeros((ab.NPLANES, case["nx2"] + 2 * NG, case["nx1"] + 2 * NG), dtype=torch.float64, device=drho.device)
    inner = D[:, NG:-NG, NG:-NG]
    inner[0], inner[1], inner[2], inner[4] = drho, 2.0 * drho, drho, 2.5 * drho
    return D


# ---------------------------------------------------------------------------
# the same values in plain torch
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "ensemble":
        items = _instances(case)
        order = sorted(range(case["n"]), key=lambda k: items[k]["nx1"] * items[k]["nx2"])
        few = set(order[:max(1, int(10.0 / (EXACT_STATE_SECONDS * case["steps"])))])
        states = [None] * case["n"]
        for k in few:
            states[k] = _exact_march(items[k], seed, case["steps"])[0]
        return {"states": states, "dt": None, "time": None}
    if case["kind"] in ("march", "dropin"):
        S, dt, time = _exact_march(case, seed, case["steps"])
        return {"state": S, "dt": dt, "time": time}
    J, g = _exact_gradient(case, seed)
    if case["kind"] == "gradient":
        return {"J": J, "gradient": g}
    return {"J": J, "dJ": float((g * _direction(case, seed)).sum()), "dS": None}


def _exact_march(case, seed, steps):
    box = _Box(case)
    with torch.no_grad():
        S = box.fill(_initial(case, seed))
        dt = COUR / box.rate(S)
        time = 0.0
        for _ in range(steps):
            S = box.fill(box.step(S, dt))
            time += float(dt)
            dt = _lesser(2.0 * dt, COUR / box.rate(S))
    return S, float(dt), time


def _exact_gradient(case, seed):
    box = _Box(case)
    S0 = _initial(case, seed).requires_grad_(True)

    def advance(S, dt):
        S = box.fill(box.step(S, dt))
        return S, _lesser(2.0 * dt, COUR / box.rate(S))

    S = box.fill(S0)
    dt = COUR / box.rate(S)
    for _ in range(case["steps"]):
        S, dt = checkpoint(advance, S, dt, use_reentrant=False)
    inner = S[:, NG:-NG, NG:-NG]
    J = (0.5 * (inner[5] ** 2 + inner[6] ** 2)).sum()
    (g,) = torch.autograd.grad(J, S0)
    return float(J), g


def _lesser(a, b):
    return torch.where(a < b, a, b)


def _greater(a, b):
    return torch.where(a > b, a, b)


def _root(x):
    """Square root whose derivative at zero is zero."""
    on = x > 0.0
    return torch.where(on, torch.sqrt(torch.where(on, x, torch.ones_like(x))), torch.zeros_like(x))


def _over(a, b, on):
    """a / b where `on`, else 0 (with no derivative there)."""
    return torch.where(on, a / torch.where(on, b, torch.ones_like(b)), torch.zeros_like(a))


class _Box:
    """The scheme on one grid's geometry: planes in the framework's order."""

    def __init__(self, case):
        x1min, x1max, x2min, x2max = _box(case)
        self.nx1, self.nx2 = case["nx1"], case["nx2"]
        self.dx1, self.dx2 = (x1max - x1min) / case["nx1"], (x2max - x2min) / case["nx2"]
        self.bc, self.hlle = _bc(case), case["flux"] == "hlle"

    # ghost zones -----------------------------------------------------------
    def _sources(self, n, inner, outer, face):
        """Index and sign from which each entry along one direction is taken."""
        src, flip = list(range(n + 2 * NG)), [False] * (n + 2 * NG)
        first, last = NG, NG + n - 1
        for k in range(1, NG + 1):
            src[first - k] = {1: first + k - 1, 2: first, 4: last - k + 1}[inner]
            flip[first - k] = inner == 1
            if not (face and k == 1):   # the face beyond the last cell is the step's own
                src[last + k] = {1: last - (k - 2 if face else k - 1), 2: last, 4: first + k - 1}[outer]
                flip[last + k] = outer == 1
        return src, flip

    def fill(self, S):
        planes = list(S)
        for axis, n, (inner, outer), normal_face, momentum in ((1, self.nx1, self.bc[:2], 8, 1),
                                                               (0, self.nx2, self.bc[2:], 9, 2)):
            for p in range(ab.NPLANES):
                src, flip = self._sources(n, inner, outer, p == normal_face)
                a = planes[p].index_select(axis, torch.tensor(src, device=S.device))
                if p == momentum and any(flip):
                    sign = torch.tensor([-1.0 if f else 1.0 for f in flip], dtype=S.dtype, device=S.device)
                    a = a * (sign[None, :] if axis == 1 else sign[:, None])
                if axis == 1:   # x1 ghosts belong to interior rows; x2 then copies whole rows
                    rows = self.nx2 + (1 if p == 9 else 0)
                    a = torch.cat([planes[p][:NG], a[NG:NG + rows], planes[p][NG + rows:]])
                planes[p] = a
        return torch.stack(planes)

    def rate(self, S):
        d, m1, m2, m3, e = (S[p, NG:-NG, NG:-NG] for p in range(5))
        v1, v2, v3 = m1 / d, m2 / d, m3 / d
        p = (GAMMA - 1.0) * (e - 0.5 * d * (v1 * v1 + v2 * v2 + v3 * v3))
        ca = _root(GAMMA * torch.clamp(p, min=1.0e-20) / d)
        r = _greater((v1.abs() + ca) / self.dx1, (v2.abs() + ca) / self.dx2).flatten()
        return r[torch.argmax(r.detach())]

    # one step --------------------------------------------------------------
    def step(self, S, dt):
        def east(a, k=1):
            return torch.roll(a, -k, 1)

        def north(a, k=1):
            return torch.roll(a, -k, 0)

        d, M1, M2, M3, E, B1c, B2c, B3c, B1i, B2i, _ = S
        q1, q2 = dt / self.dx1, dt / self.dx2
        h1, h2 = 0.5 * q1, 0.5 * q2
        # predictor states and fluxes of both sweeps, in the sweep's frame
        wl, wr = _plm(_primitive((d, M1, M2, M3, E, B2c, B3c), B1c), B1c, q1, east)
        src = 0.5 * dt * (M2 / d) * (east(B1i) - B1i) / self.dx1
        wl[5], wr[5] = wl[5] + src, wr[5] + src
        wl = [east(a, -1) for a in wl]
        ulx, urx = _conserved(wl, B1i), _conserved(wr, B1i)
        fx = self._riemann(ulx, urx, wl, wr, B1i)
        wl, wr = _plm(_primitive((d, M2, M3, M1, E, B3c, B1c), B2c), B2c, q2, north)
        src = 0.5 * dt * (M1 / d) * (north(B2i) - B2i) / self.dx2
        wl[6], wr[6] = wl[6] + src, wr[6] + src
        wl = [north(a, -1) for a in wl]
        uly, ury = _conserved(wl, B2i), _conserved(wr, B2i)
        fy = self._riemann(uly, ury, wl, wr, B2i)
        emf = _corner(fx, fy, (B1c * M2 - B2c * M1) / d, east, north)
        # half-step face fields, transverse corrections, corrector fluxes
        B1h, B2h = B1i - h2 * (north(emf) - emf), B2i + h1 * (east(emf) - emf)
        gy = [h2 * (north(f) - f) for f in fy]   # d, M2, M3, M1, E, B3, B1
        tx = [gy[0], gy[3], gy[1], gy[2], gy[4], None, gy[5]]
        ul, ur = _minus(ulx, [a if a is None else east(a, -1) for a in tx]), _minus(urx, tx)
        add = _source(h1 * (east(B1i) - B1i), (B1c, B2c, B3c), M3 / d, E)
        ul = [u + a for u, a in zip(ul, [east(a, -1) for a in add])]
        ur = [u + a for u, a in zip(ur, add)]
        fx2 = self._riemann(ul, ur, _primitive(ul, B1h), _primitive(ur, B1h), B1h)
        gx = [h1 * (east(f) - f) for f in fx]    # d, M1, M2, M3, E, B2, B3
        ty = [gx[0], gx[2], gx[3], gx[1], gx[4], gx[6], None]
        ul, ur = _minus(uly, [a if a is None else north(a, -1) for a in ty]), _minus(ury, ty)
        a = _source(h2 * (north(B2i) - B2i), (B2c, B3c, B1c), M3 / d, E, v3_slot=1, v3_field=1)
        ul = [u + b for u, b in zip(ul, [north(b, -1) for b in a])]
        ur = [u + b for u, b in zip(ur, a)]
        fy2 = self._riemann(ul, ur, _primitive(ul, B2h), _primitive(ur, B2h), B2h)
        # half-step cell EMF, then the full update
        dh = d - gx[0] - gy[0]
        m1, m2 = M1 - gx[1] - gy[3], M2 - gx[2] - gy[1]
        b1, b2 = 0.5 * (B1h + east(B1h)), 0.5 * (B2h + north(B2h))
        emf = _corner(fx2, fy2, (b1 * m2 - b2 * m1) / dh, east, north)
        B1n, B2n = B1i - q2 * (north(emf) - emf), B2i + q1 * (east(emf) - emf)
        dx = [q1 * (east(f) - f) for f in fx2]
        dy = [q2 * (north(f) - f) for f in fy2]
        B3n = B3c - dx[6] - dy[5]
        return torch.stack([d - dx[0] - dy[0], M1 - dx[1] - dy[3], M2 - dx[2] - dy[1], M3 - dx[3] - dy[2],
                            E - dx[4] - dy[4], 0.5 * (B1n + east(B1n)), 0.5 * (B2n + north(B2n)), B3n,
                            B1n, B2n, B3n])

    # fluxes ----------------------------------------------------------------
    def _riemann(self, ul, ur, wl, wr, bn):
        rl, rr = _root(wl[0]), _root(wr[0])
        isum = 1.0 / (rl + rr)
        d = rl * rr
        v1, v2, v3 = ((rl * wl[n] + rr * wr[n]) * isum for n in (1, 2, 3))
        b2, b3 = ((rr * wl[n] + rl * wr[n]) * isum for n in (5, 6))
        xf = 0.5 * ((wl[5] - wr[5]) ** 2 + (wl[6] - wr[6]) ** 2) * isum * isum
        yf = 0.5 * (wl[0] + wr[0]) / d
        pl, pr = (0.5 * (bn * bn + w[5] ** 2 + w[6] ** 2) for w in (wl, wr))
        h = ((ul[4] + wl[4] + pl) / rl + (ur[4] + wr[4] + pr) / rr) * isum
        vsq, btsq = v1 * v1 + v2 * v2 + v3 * v3, b2 * b2 + b3 * b3
        gf = (GAMMA - 1.0) - (GAMMA - 2.0) * yf
        vax2 = bn * bn / d
        hp = h - (vax2 + btsq / d)
        a2 = torch.clamp((GAMMA - 1.0) * (hp - 0.5 * vsq) - (GAMMA - 2.0) * xf, min=1.0e-20)
        ct2 = gf * btsq / d
        disc = _root((vax2 + ct2 - a2) ** 2 + 4.0 * a2 * ct2)
        cf2 = 0.5 * (vax2 + ct2 + a2 + disc)
        cs2 = a2 * vax2 / cf2
        cf, cs, va = _root(cf2), _root(cs2), _root(vax2)
        hlle = self._hlle(ul, ur, wl, wr, bn, pl, pr, v1 - cf, v1 + cf)
        if self.hlle:
            return hlle
        ev = [v1 - cf, v1 - va, v1 - cs, v1, v1 + cs, v1 + va, v1 + cf]
        fl, fr = _side_flux(ul, wl, bn, pl), _side_flux(ur, wr, bn, pr)
        # eigenvectors of the Roe matrix (adiabatic MHD, Cargo & Gallice)
        s = torch.where(bn < 0.0, -1.0, 1.0).to(bn.dtype)
        bt = _root(btsq)
        e2, e3 = _unit(b2, b3, bt, btsq, bn * bn + d * a2)
        sg = _root(gf)
        e2s, e3s = e2 / sg, e3 / sg
        ess = e2s * e2s + e3s * e3s
        bts = _root(gf * btsq)
        af, as_ = _alphas(cf2 - cs2, a2 - cs2, cf2 - a2)
        rd, a = _root(d), _root(a2)
        qf, qs = cf * af * s, cs * as_ * s
        afp, asp = a * af / rd, a * as_ / rd
        vb, vq = v2 * e2s + v3 * e3s, (v2 * e2s + v3 * e3s) / ess
        gx = (GAMMA - 2.0) * xf / (GAMMA - 1.0)
        zero = torch.zeros_like(d)
        R = [
            [af, af * ev[0], af * v2 + qs * e2s, af * v3 + qs * e3s,
             af * (hp - v1 * cf) + qs * vb + asp * bts * ess, asp * e2s, asp * e3s],
            [zero, zero, -e3, e2, -(v2 * e3 - v3 * e2), -e3 * s / rd, e2 * s / rd],
            [as_, as_ * ev[2], as_ * v2 - qf * e2s, as_ * v3 - qf * e3s,
             as_ * (hp - v1 * cs) - qf * vb - afp * bts * ess, -afp * e2s, -afp * e3s],
            [torch.ones_like(d), v1, v2, v3, 0.5 * vsq + gx, zero, zero],
            [as_, as_ * ev[4], as_ * v2 + qf * e2s, as_ * v3 + qf * e3s,
             as_ * (hp + v1 * cs) + qf * vb - afp * bts * ess, -afp * e2s, -afp * e3s],
            [zero, zero, e3, -e2, v2 * e3 - v3 * e2, -e3 * s / rd, e2 * s / rd],
            [af, af * ev[6], af * v2 - qs * e2s, af * v3 - qs * e3s,
             af * (hp + v1 * cf) - qs * vb + asp * bts * ess, asp * e2s, asp * e3s],
        ]
        n = 0.5 / a2
        cff, css, qfn, qsn = n * af * cf, n * as_ * cs, n * qf, n * qs
        AF, AS, afb, asb = n * afp * d, n * asp * d, n * afp * bts, n * asp * bts
        afn, asn = n * (GAMMA - 1.0) * af, n * (GAMMA - 1.0) * as_
        n2 = 2.0 * n * (GAMMA - 1.0)
        q2, q3, vh = e2s / ess, e3s / ess, vsq - hp

        def fast(g):   # g = +1 for the left-going fast wave
            return [afn * vh + cff * (cf + g * v1) - g * qsn * vq - asb, -afn * v1 - g * cff,
                    -afn * v2 + g * qsn * q2, -afn * v3 + g * qsn * q3, afn, AS * q2 - afn * b2, AS * q3 - afn * b3]

        def slow(g):
            return [asn * vh + css * (cs + g * v1) + g * qfn * vq + afb, -asn * v1 - g * css,
                    -asn * v2 - g * qfn * q2, -asn * v3 - g * qfn * q3, asn, -AF * q2 - asn * b2, -AF * q3 - asn * b3]

        def alfven(g):
            return [g * 0.5 * (v2 * e3 - v3 * e2), zero, -g * 0.5 * e3, g * 0.5 * e2, zero,
                    -0.5 * rd * e3 * s, 0.5 * rd * e2 * s]

        entropy = [1.0 - n2 * (0.5 * vsq - gx), n2 * v1, n2 * v2, n2 * v3, -n2, n2 * b2, n2 * b3]
        L = [fast(1.0), alfven(1.0), slow(1.0), entropy, slow(-1.0), alfven(-1.0), fast(-1.0)]
        du = [r - q for r, q in zip(ur, ul)]
        amp = [sum(L[k][m] * du[m] for m in range(7)) for k in range(7)]
        F = [0.5 * (p + q) for p, q in zip(fl, fr)]
        u, bad = list(ul), torch.zeros_like(d, dtype=torch.bool)
        for k in range(7):
            F = [f - 0.5 * ev[k].abs() * amp[k] * R[k][m] for m, f in enumerate(F)]
            if k < 6:
                u = [(q + amp[k] * R[k][m]).detach() for m, q in enumerate(u)]
                p = u[4] - 0.5 * (u[1] ** 2 + u[2] ** 2 + u[3] ** 2) / u[0] - 0.5 * (u[5] ** 2 + u[6] ** 2 + bn * bn)
                bad = bad | ((ev[k + 1] > ev[k]) & ((u[0] <= 0.0) | (p < 0.0)))
        out = []
        for m in range(7):
            f = torch.where(bad, hlle[m], F[m])
            f = torch.where(ev[6] <= 0.0, fr[m], f)
            out.append(torch.where(ev[0] >= 0.0, fl[m], f))
        return out

    @staticmethod
    def _hlle(ul, ur, wl, wr, bn, pl, pr, first, last):
        def speed(u, w):
            a2, va2, ct2 = GAMMA * w[4] / w[0], bn * bn / w[0], (u[5] ** 2 + u[6] ** 2) / w[0]
            return _root(0.5 * (va2 + ct2 + a2 + _root((va2 + ct2 - a2) ** 2 + 4.0 * a2 * ct2)))

        zero = torch.zeros_like(bn)
        bp = _greater(_greater(last, wr[1] + speed(ur, wr)), zero)
        bm = _lesser(_lesser(first, wl[1] - speed(ul, wl)), zero)
        fl = [f - bm * u for f, u in zip(_side_flux(ul, wl, bn, pl), ul)]
        fr = [f - bp * u for f, u in zip(_side_flux(ur, wr, bn, pr), ur)]
        t = 0.5 * (bp + bm) / (bp - bm)
        return [0.5 * (a + b) + (a - b) * t for a, b in zip(fl, fr)]


def _primitive(u, bn):
    d, mx, my, mz, e, by, bz = u
    p = (GAMMA - 1.0) * (e - 0.5 * (mx * mx + my * my + mz * mz) / d - 0.5 * (bn * bn + by * by + bz * bz))
    return [d, mx / d, my / d, mz / d, torch.clamp(p, min=1.0e-20), by, bz]


def _conserved(w, bn):
    d, vx, vy, vz, p, by, bz = w
    e = p / (GAMMA - 1.0) + 0.5 * d * (vx * vx + vy * vy + vz * vz) + 0.5 * (bn * bn + by * by + bz * bz)
    return [d, d * vx, d * vy, d * vz, e, by, bz]


def _side_flux(u, w, bn, pb):
    d, vx, vy, vz, p, by, bz = w
    return [u[1], u[1] * vx + p - 0.5 * (bn * bn - by * by - bz * bz), u[1] * vy - bn * by, u[1] * vz - bn * bz,
            (u[4] + p) * vx + pb * vx - bn * (bn * vx + by * vy + bz * vz), by * vx - bn * vy, bz * vx - bn * vz]


def _minus(u, g):
    return [a if b is None else a - b for a, b in zip(u, g)]


def _source(db, b, v3, like, v3_slot=3, v3_field=2):
    """MHD source terms of the transverse correction in the sweep's frame:
    b = (normal, second, third) fields, the out-of-plane one at v3_field."""
    zero = torch.zeros_like(like)
    out = [zero, db * b[0], db * b[1], db * b[2], db * b[v3_field] * v3, zero, zero]
    out[6 if v3_slot == 3 else 5] = db * v3
    return out


def _alphas(span, slow_gap, fast_gap):
    """Renormalisation coefficients of the fast and slow waves."""
    one, zero = torch.ones_like(span), torch.zeros_like(span)
    mid = (span != 0.0) & (slow_gap > 0.0) & (fast_gap > 0.0)
    af, as_ = _root(_over(slow_gap, span, mid)), _root(_over(fast_gap, span, mid))
    only_slow = (span != 0.0) & (slow_gap <= 0.0)
    return (torch.where(mid, af, torch.where(only_slow, zero, one)),
            torch.where(mid, as_, torch.where(only_slow, one, zero)))


def _unit(b2, b3, bt, btsq, scale):
    """Direction of the transverse field: (1, 0) where it vanishes, and
    constant under differentiation where it is negligible."""
    on = bt != 0.0
    e2 = torch.where(on, _over(b2, bt, on), torch.ones_like(bt))
    e3 = _over(b3, bt, on)
    frozen = btsq < 1.0e-12 * scale
    return torch.where(frozen, e2.detach(), e2), torch.where(frozen, e3.detach(), e3)


def _plm(w, bn, dtodx, ahead):
    """Characteristic piecewise linear states: (left state of each cell's
    outer face, right state of its inner face) after half a step."""
    d, v1, _, _, p, b2, b3 = w
    di, btsq, a2 = 1.0 / d, b2 * b2 + b3 * b3, GAMMA * p / d
    va2, ct2 = bn * bn * di, btsq * di
    disc = _root((va2 + ct2 - a2) ** 2 + 4.0 * a2 * ct2)
    cf2 = 0.5 * (va2 + ct2 + a2 + disc)
    cs2 = a2 * va2 / cf2
    cf, cs, va, a, rd = _root(cf2), _root(cs2), _root(va2), _root(a2), _root(d)
    e2, e3 = _unit(b2, b3, _root(btsq), btsq, bn * bn + d * a2)
    af, as_ = _alphas(disc, a2 - cs2, cf2 - a2)
    s = torch.where(bn < 0.0, -1.0, 1.0).to(bn.dtype)
    qf, qs, AF, AS = cf * af * s, cs * as_ * s, a * af * rd, a * as_ * rd
    zero, one, n = torch.zeros_like(d), torch.ones_like(d), 0.5 / a2
    ev = [v1 - cf, v1 - va, v1 - cs, v1, v1 + cs, v1 + va, v1 + cf]

    def fast(g):
        return ([d * af, -g * cf * af, g * qs * e2, g * qs * e3, d * a2 * af, AS * e2, AS * e3],
                [zero, -g * n * cf * af, g * n * qs * e2, g * n * qs * e3, n * af * di, n * AS * di * e2,
                 n * AS * di * e3])

    def slow(g):
        return ([d * as_, -g * cs * as_, -g * qf * e2, -g * qf * e3, d * a2 * as_, -AF * e2, -AF * e3],
                [zero, -g * n * cs * as_, -g * n * qf * e2, -g * n * qf * e3, n * as_ * di, -n * AF * di * e2,
                 -n * AF * di * e3])

    def alfven(g):
        return ([zero, zero, -g * e3, g * e2, zero, -e3 * s * rd, e2 * s * rd],
                [zero, zero, -g * 0.5 * e3, g * 0.5 * e2, zero, -0.5 * e3 * s / rd, 0.5 * e2 * s / rd])

    entropy = ([one, zero, zero, zero, zero, zero, zero], [one, zero, zero, zero, -1.0 / a2, zero, zero])
    waves = [fast(1.0), alfven(1.0), slow(1.0), entropy, slow(-1.0), alfven(-1.0), fast(-1.0)]
    R, L = [r for r, _ in waves], [q for _, q in waves]
    dl, dr = [q - ahead(q, -1) for q in w], [ahead(q) - q for q in w]
    dc = [ahead(q) - ahead(q, -1) for q in w]
    dg = [_over(2.0 * x * y, x + y, x * y > 0.0) for x, y in zip(dl, dr)]
    slope = [zero] * 7
    for k in range(7):
        c, l, r, g = (sum(L[k][m] * q[m] for m in range(7)) for q in (dc, dl, dr, dg))
        lim = _lesser(2.0 * _lesser(l.abs(), r.abs()), _lesser(0.5 * c.abs(), g.abs()))
        da = torch.where(l * r > 0.0, torch.where(c < 0.0, -lim, lim), zero)
        slope = [q + da * R[k][m] for m, q in enumerate(slope)]
    wl, wr, dw = [], [], []
    for q, g in zip(w, slope):
        back, fore = ahead(q, -1), ahead(q)
        lo = _lesser(_greater(q, back), _greater(_lesser(q, back), q - 0.5 * g))
        hi = _lesser(_greater(q, fore), _greater(_lesser(q, fore), q + 0.5 * g))
        wl.append(lo), wr.append(hi), dw.append(hi - lo)
    pl = [q - 0.5 * _greater(ev[6], zero) * dtodx * g for q, g in zip(wr, dw)]
    pr = [q - 0.5 * _lesser(ev[0], zero) * dtodx * g for q, g in zip(wl, dw)]
    for k in range(7):
        strength = sum(L[k][m] * dw[m] for m in range(7)) * 0.5 * dtodx
        to_left = torch.where(ev[k] != 0.0, strength * (ev[6] - ev[k]), zero)
        to_right = torch.where(ev[k] < 0.0, strength * (ev[0] - ev[k]), zero)
        pl = [q + to_left * R[k][m] for m, q in enumerate(pl)]
        pr = [q + to_right * R[k][m] for m, q in enumerate(pr)]
    return pl, pr


def _corner(fx, fy, cell, east, north):
    """Upwind corner EMF from the face fluxes and the cell EMF."""
    ex, ey = -fx[5], fy[6]
    ex_s, ey_w = north(ex, -1), east(ey, -1)
    c_s, c_w = north(cell, -1), east(cell, -1)
    c_sw = north(c_w, -1)

    def pick(flow, behind, ahead):
        return torch.where(flow > 0.0, behind, torch.where(flow < 0.0, ahead, 0.5 * (behind + ahead)))

    l2 = ex_s + pick(north(fx[0], -1), ey_w - c_sw, ey - c_s)
    r2 = ex + pick(fx[0], ey_w - c_w, ey - cell)
    l1 = ey_w + pick(east(fy[0], -1), ex_s - c_sw, ex - c_w)
    r1 = ey + pick(fy[0], ex_s - c_s, ex - cell)
    return 0.25 * (l1 + r1 + l2 + r2)
