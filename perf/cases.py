"""Workloads of the framework's public entry points, for timing and for checking
results: listed() and draw() say which, prepare() makes what a program has in hand
before the call, run() is one pass, work() what a pass cannot do without, exact()
the same results in plain torch in 64 bits.

Kinds (every one through an entry point that a user's program calls):
  solver    a state tensor is loaded (Solver.put_state) and advanced by `steps` TVD-RK2
            steps of the fused kernels: 2D and 3D, FP64 and FP32-mixed
  host      the same with the state in page-locked host memory on both sides
            (Solver.step_host), as a host code that calls the library once per step
  ensemble  independent 2D grids of different sizes advanced together (Ensemble)
  adjoint   forward run and gradient of it (adjoint.Evolve under torch autograd)
  routines  one step built from the reference-named routines on device arrays, as
            a driver that replaces its own routines one by one makes it
"""
import math

import torch

from openmhd_gb300 import Solver, field_loop3d, harris3d, kelvin_helmholtz, orszag_tang, reconnection2d
from openmhd_gb300 import routines
from openmhd_gb300.solver import ModelSpec

MX, MY, MZ, EN, RO, BX, BY, BZ, PS = range(9)
VX, VY, VZ, PR = range(4)


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the smallest grids: parameter scans and tests, bound by the latency of one step
        {"name": "ot-64x64-fp64", "kind": "solver", "problem": "ot", "nx": 64, "ny": 64, "nz": 0, "limiter": "mc",
         "precision": "fp64", "steps": 10},
        # the reference's Orszag-Tang vortex at the size its driver is set to
        {"name": "ot-256x256-fp64", "kind": "solver", "problem": "ot", "nx": 256, "ny": 256, "nz": 0, "limiter": "mc",
         "precision": "fp64", "steps": 10},
        # an odd-sized grid with walls, called once per step from a host code
        {"name": "kh-host-999x501-fp64", "kind": "host", "problem": "kh", "nx": 999, "ny": 501, "nz": 0,
         "limiter": "minmod", "precision": "fp64", "steps": 1},
        # the benchmark's grid, in both precisions
        {"name": "kh-4096x2048-fp64", "kind": "solver", "problem": "kh", "nx": 4096, "ny": 2048, "nz": 0,
         "limiter": "minmod", "precision": "fp64", "steps": 2},
        {"name": "kh-4096x2048-mixed", "kind": "solver", "problem": "kh", "nx": 4096, "ny": 2048, "nz": 0,
         "limiter": "minmod", "precision": "mixed", "steps": 3},
        # resistive 2D reconnection between symmetry walls, a quarter of the reference's resolution
        {"name": "recon2d-500x125-fp64", "kind": "solver", "problem": "recon2d", "nx": 500, "ny": 125, "nz": 0,
         "limiter": "minmod", "precision": "fp64", "steps": 5},
        # a parameter study: grids of different sizes and boundaries in one batch
        {"name": "ensemble-24-mixed", "kind": "ensemble", "problem": "mix", "members": 24, "side_lo": 128,
         "side_hi": 512, "precision": "mixed", "steps": 10},
        # resistive 3D Harris sheet: a small run and a production-sized one
        {"name": "harris-64x32x64-fp64", "kind": "solver", "problem": "harris", "nx": 64, "ny": 32, "nz": 64,
         "limiter": "mc", "precision": "fp64", "steps": 3},
        {"name": "harris-256x128x256-mixed", "kind": "solver", "problem": "harris", "nx": 256, "ny": 128, "nz": 256,
         "limiter": "mc", "precision": "mixed", "steps": 2},
        # the reference's 3D field-loop advection at the size its driver is set to
        {"name": "loop-100x100x200-fp64", "kind": "solver", "problem": "loop", "nx": 100, "ny": 100, "nz": 200,
         "limiter": "minmod", "precision": "fp64", "steps": 2},
        # gradient of a Kelvin-Helmholtz run with respect to its initial state
        {"name": "adjoint-512x256", "kind": "adjoint", "problem": "kh", "nx": 512, "ny": 256, "nz": 0,
         "limiter": "minmod", "precision": "fp64", "steps": 12, "every": 4},
        # one step through the routine-level drop-ins
        {"name": "routines-1024x512", "kind": "routines", "problem": "ot", "nx": 1024, "ny": 512, "nz": 0,
         "limiter": "mc", "precision": "fp64", "steps": 1},
    ]


def draw(rng):
    def size(lo, hi):  # spread over the logarithm, odd ones among them
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["2d", "2d", "2d", "3d", "3d", "host", "ensemble", "adjoint", "routines"])
    limiter = rng.choice(["minmod", "mc"])
    if kind == "3d":
        precision = rng.choice(["fp64", "mixed"])
        big = 6.0e6 if precision == "mixed" else 1.8e6  # interior cells
        if rng.random() < 0.5:  # resistive: equal spacings, ny = nx / 2
            ny = size(16, 88)
            nx = 2 * ny
            nz = nx
            problem = "harris"
        else:
            nx, ny, nz = size(24, 180), size(24, 180), size(24, 240)
            problem = "loop"
        cells = nx * ny * nz
        if cells > big:
            nz = max(24, int(nz * big / cells)) if problem == "loop" else nz
        return {"kind": "solver", "problem": problem, "nx": nx, "ny": ny, "nz": nz, "limiter": limiter,
                "precision": precision, "steps": 2}
    if kind == "ensemble":
        return {"kind": "ensemble", "problem": "mix", "members": rng.randint(2, 30), "side_lo": 128,
                "side_hi": size(160, 512), "precision": rng.choice(["mixed", "mixed", "fp64"]),
                "steps": rng.randint(3, 10)}
    if kind == "adjoint":
        return {"kind": "adjoint", "problem": "kh", "nx": size(64, 640), "ny": size(48, 320), "nz": 0,
                "limiter": limiter, "precision": "fp64", "steps": rng.randint(5, 12), "every": rng.randint(2, 5)}
    if kind == "routines":
        return {"kind": "routines", "problem": rng.choice(["ot", "kh"]), "nx": size(64, 2048), "ny": size(64, 1024),
                "nz": 0, "limiter": limiter, "precision": "fp64", "steps": 1}
    if kind == "host":
        return {"kind": "host", "problem": rng.choice(["ot", "kh"]), "nx": size(128, 2048), "ny": size(128, 1024),
                "nz": 0, "limiter": limiter, "precision": rng.choice(["fp64", "mixed"]), "steps": 1}
    problem = rng.choice(["ot", "kh", "kh", "recon2d"])
    precision = rng.choice(["fp64", "fp64", "mixed"])
    nx, ny = size(48, 3000), size(48, 2000)
    if problem == "recon2d":
        nx, ny = size(64, 1200), size(48, 400)
    return {"kind": "solver", "problem": problem, "nx": nx, "ny": ny, "nz": 0, "limiter": limiter,
            "precision": precision, "steps": 2 if nx * ny > 500000 else 6}


def _config(case):
    """The framework's own problem set-up of a case."""
    cfg = _setup(case)
    if case["kind"] == "routines":  # the reference's routines take one spacing
        cfg.dy = cfg.dx
    return cfg


def _setup(case):
    k = {"precision": case["precision"], "limiter": case["limiter"]}
    p = case["problem"]
    if p == "ot":
        return orszag_tang(case["nx"], case["ny"], **k)[0]
    if p == "kh":
        return kelvin_helmholtz(case["nx"], case["ny"], **k)[0]
    if p == "recon2d":
        return reconnection2d(case["nx"], case["ny"], **k)[0]
    if p == "harris":
        return harris3d(case["nx"], case["ny"], case["nz"], **k)[0]
    return field_loop3d(case["nx"], case["ny"], case["nz"], **k)[0]


def _members(case, seed):
    """Configurations and models of an ensemble: half Orszag-Tang, half Kelvin-Helmholtz,
    the sizes spread over the sides of the case, the rest from the seed."""
    g = torch.Generator().manual_seed(seed)
    u = lambda lo, hi: lo + (hi - lo) * float(torch.rand((), generator=g, dtype=torch.float64))  # noqa: E731
    sizes = torch.Generator().manual_seed(case["members"])  # the sizes are the case's, not the seed's
    cfgs, models = [], []
    for i in range(case["members"]):
        side = torch.randint(case["side_lo"] // 32, case["side_hi"] // 32 + 1, (2,), generator=sizes)
        nx, ny = (32 * int(v) for v in side)
        if i % 2 == 0:
            c, m = orszag_tang(nx, ny, precision=case["precision"], amp=u(0.5, 1.5), phase_x=u(0, 2 * math.pi),
                               phase_y=u(0, 2 * math.pi))
        else:
            c, m = kelvin_helmholtz(nx, ny, precision=case["precision"], shear=u(0.3, 0.8), bx0=u(0.05, 0.3),
                                    seed=int(u(0, 2 ** 31)))
        cfgs.append(c)
        models.append(m)
    return cfgs, models


# --------------------------------------------------------------------------
# initial states, (9, [nz + 2,] ny + 2, nx + 2) in 64 bits with the ghost cells set
# --------------------------------------------------------------------------
def _axes(cfg):
    out = []
    for n, d, x0 in ((cfg.ix, cfg.dx, cfg.x0), (cfg.jx, cfg.dy, cfg.y0), (cfg.kx, cfg.dz, cfg.z0)):
        out.append(x0 - d / 2 + d * torch.arange(n, device="cuda", dtype=torch.float64))
    x, y, z = out
    return (x[None, :], y[:, None], None) if cfg.nd == 2 else (x[None, None, :], y[None, :, None], z[:, None, None])


def _modes(cfg, ax, g, count=3):
    """A smooth field of order one: a few periodic modes with random phases."""
    ext = (cfg.dx * (cfg.ix - 2), cfg.dy * (cfg.jx - 2), cfg.dz * (cfg.kx - 2))
    f = 0.0
    for _ in range(count):
        arg = 2 * math.pi * float(torch.rand((), generator=g, dtype=torch.float64))
        for a, e in zip(ax, ext):
            if a is not None:
                arg = arg + 2 * math.pi * int(torch.randint(1, 4, (), generator=g)) * a / e
        f = f + torch.sin(arg) / count
    return f


def _conserved(cfg, ro, v, p, B, psi=0.0):
    shape = cfg.shape[1:]
    t = [torch.broadcast_to(torch.as_tensor(a, device="cuda", dtype=torch.float64), shape) for a in (ro, *v, p, *B, psi)]
    ro, vx, vy, vz, p, bx, by, bz, psi = t
    en = 0.5 * (ro * (vx * vx + vy * vy + vz * vz) + bx * bx + by * by + bz * bz) + p / (cfg.gamma - 1)
    return _fill(torch.stack([ro * vx, ro * vy, ro * vz, en, ro, bx, by, bz, psi]), cfg)


def _initial(case, seed):
    cfg = _config(case)
    g = torch.Generator().manual_seed(seed)
    ax = _axes(cfg)
    x, y, z = ax
    m = lambda: _modes(cfg, ax, g)  # noqa: E731
    if case["problem"] == "ot":
        px, py = (2 * math.pi * float(v) for v in torch.rand(2, generator=g, dtype=torch.float64))
        return cfg, _conserved(cfg, cfg.gamma ** 2, (-torch.sin(y + py), torch.sin(x + px), 0.0), cfg.gamma,
                               (-torch.sin(y + py), torch.sin(2 * (x + px)), 0.0))
    if case["problem"] == "kh":
        # the shear layer, its noise and, as in a run that is under way, weak large-scale modes in every variable
        noise = torch.rand(cfg.shape[1:], generator=torch.Generator("cuda").manual_seed(seed), device="cuda",
                           dtype=torch.float64) * 2 - 1
        vy = 0.01 * torch.exp(-y * y) * (noise if case["kind"] != "adjoint" else m())
        e = 0.02
        return cfg, _conserved(cfg, 1 + e * m(), (0.5 * torch.tanh(y) + e * m(), vy + e * m(), e * m()),
                               0.5 * (1 + e * m()), (0.2 + e * m(), e * m(), e * m()), 0.01 * m())
    if case["problem"] == "recon2d":
        ch2 = 1 / torch.cosh(torch.clamp(y, max=25.0)) ** 2
        ro = 1 + ch2 / 0.2
        ex = torch.exp(-(x * x + y * y) / 4)
        b1 = 0.03 * (1 + 0.2 * float(torch.rand((), generator=g, dtype=torch.float64)))
        return cfg, _conserved(cfg, ro, (0.01 * m(), 0.01 * m(), 0.01 * m()), 0.1 * ro,
                               (torch.tanh(y) - b1 * y * ex, b1 * x * ex, 0.01 * m()))
    if case["problem"] == "harris":
        ro = 1 + 1 / torch.cosh(z) ** 2 / 0.2
        near = 0.01 * torch.exp(-z * z / 4)
        return cfg, _conserved(cfg, ro, (near * m(), near * m(), near * m()), 0.1 * ro,
                               (torch.tanh(z) + near * m(), near * m(), near * m()))
    # field loop: uniform flow, a weak field with a sharp edge, carried across the grid
    a = torch.clamp(0.3 - torch.sqrt(y * y + ((2 * x + z + 0.2 * m()) ** 2) / 5), min=0.0)
    e = 1e-3
    return cfg, _conserved(cfg, 1 + e * m(), (1 + e * m(), 1 + e * m(), 2 + e * m()), 1 + e * m(),
                           (e * torch.gradient(a, dim=1)[0] / cfg.dy, e * m(), e * torch.gradient(a, dim=0)[0] / cfg.dz))


# --------------------------------------------------------------------------
# prepare and run
# --------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "ensemble":
        from openmhd_gb300.ensemble import Ensemble

        cfgs, models = _members(case, seed)
        ens = Ensemble(cfgs)
        # the tiling that the autotuner settles on for ensembles of this kind, set so that a run does not depend on a timing
        ens.set_tiling(*((4, 4) if case["precision"] == "mixed" else (2, 2)))
        out = [torch.empty(c.shape, dtype=torch.float64, device="cuda") for c in cfgs]
        return {"case": case, "ens": ens, "models": models, "out": out}
    cfg, U0 = _initial(case, seed)
    st = {"case": case, "cfg": cfg, "U0": U0}
    if case["kind"] == "solver":
        st["solver"] = Solver(cfg)
    elif case["kind"] == "host":
        st["solver"] = Solver(cfg)
        st["in"] = U0.cpu().pin_memory()
        st["out"] = torch.empty(cfg.shape, dtype=torch.float64, pin_memory=True)
    elif case["kind"] == "adjoint":
        from openmhd_gb300.adjoint import AdjointRun

        st["run"] = AdjointRun(cfg, case["steps"], case["every"])
        st["gUN"] = _cotangent(cfg, seed)
    else:
        new = lambda k: torch.empty((k,) + cfg.shape[1:], dtype=torch.float64, device="cuda")  # noqa: E731
        st.update(U=new(9), U1=new(9), V=new(4), VL=new(9), VR=new(9), F=new(9), G=new(9))
    return st


def _cotangent(cfg, seed):
    """dJ/dU_N of J = sum(c U_N) over the interior, c smooth."""
    g = torch.Generator().manual_seed(seed + 1)
    ax = _axes(cfg)
    c = torch.stack([torch.broadcast_to(_modes(cfg, ax, g), cfg.shape[1:]) for _ in range(9)]).contiguous()
    c[:, 0], c[:, -1], c[:, :, 0], c[:, :, -1] = 0.0, 0.0, 0.0, 0.0
    return c


def run(state):
    case = state["case"]
    if case["kind"] == "solver":
        s = state["solver"]
        s.put_state(state["U0"])
        s.step(case["steps"])
        return s.state()
    if case["kind"] == "host":
        state["solver"].step_host(state["in"], state["out"], n=case["steps"])
        return state["out"]
    if case["kind"] == "ensemble":
        import ctypes

        ens = state["ens"]
        ens.init_models(state["models"])
        ens.step(case["steps"])
        h = ctypes.c_void_p()
        for i, o in enumerate(state["out"]):  # member states stay on the device
            ens.lib.omhd_ensemble_member(ens._h, i, ctypes.byref(h))
            ens.lib.omhd_solver_get_state(h, o.data_ptr())
        return state["out"]
    if case["kind"] == "adjoint":
        from openmhd_gb300.adjoint import Evolve

        U0 = state["U0"].requires_grad_()
        UN = Evolve.apply(U0, state["run"])
        (g,) = torch.autograd.grad(UN, U0, state["gUN"])
        return [UN.detach(), g]
    return _routine_step(state)


def _routine_step(s):
    """One TVD-RK2 step as the reference's driver makes it from its routines."""
    cfg, U, U1, V, VL, VR = s["cfg"], s["U"], s["U1"], s["V"], s["VL"], s["VR"]
    lm = {"minmod": 1, "mc": 2}[cfg.limiter]
    U.copy_(s["U0"])
    routines.u2v(U, V)
    vmax, dt = routines.set_dt(U, V, cfg.dx, cfg.cfl)
    routines.glm_ss2(U, vmax, dt)
    for stage in (1, 2):
        S = U if stage == 1 else U1
        if stage == 2:
            routines.u2v(U1, V)
        for d, F in ((1, s["F"]), (2, s["G"])):
            for k in range(9):
                routines.limiter(V[k] if k < 4 else S[k], VL[k], VR[k], d, lm)
            q = 2 * (d - 1)
            routines.facefix(VL, VR, d, cfg.bc_kind[q], cfg.bc_flip[q], cfg.bc_kind[q + 1], cfg.bc_flip[q + 1])
            routines.flux_solver(F, VL, VR, vmax, d, 3)
        if stage == 1:
            routines.rk_tvd21(U, U1, s["F"], s["G"], dt=dt, dx=cfg.dx)
            routines.bc(U1, cfg.bc_kind, cfg.bc_flip)
        else:
            routines.rk_tvd22(U, U1, s["F"], s["G"], dt=dt, dx=cfg.dx)
            routines.bc(U, cfg.bc_kind, cfg.bc_flip)
    routines.glm_ss2(U, vmax, dt)
    return [U, V, s["F"], s["G"]]


def work(case):
    """State in and out once; the operations of the scheme (1838 a cell and step in 2D,
    2937 in 3D with resistivity, 2500 without; a step's gradient about twice a step)."""
    if case["kind"] == "ensemble":
        cells = sum(c.interior_cells for c in _members(case, 0)[0])
        return {"bytes": 144 * cells, "flops": 1838 * cells * case["steps"]}
    cells = case["nx"] * case["ny"] * max(1, case["nz"])
    per = 1838 if case["nz"] == 0 else 2937 if case["problem"] == "harris" else 2500
    if case["kind"] == "adjoint":
        return {"bytes": 288 * cells, "flops": 3 * per * cells * case["steps"]}
    planes = 9 + (31 if case["kind"] == "routines" else 9)
    return {"bytes": 8 * planes * cells, "flops": per * cells * case["steps"]}


# --------------------------------------------------------------------------
# the same results in plain torch, 64 bits (2D and 3D, HLLD, minmod and MC)
# --------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "ensemble":
        cfgs, models = _members(case, seed)
        return [_evolve(c, _model(c, m), case["steps"]) for c, m in zip(cfgs, models)]
    cfg, U0 = _initial(case, seed)
    if case["kind"] == "adjoint":
        U0.requires_grad_()
        UN = _evolve(cfg, U0, case["steps"])
        (g,) = torch.autograd.grad(UN, U0, _cotangent(cfg, seed))
        return [UN.detach(), g]
    with torch.no_grad():
        if case["kind"] == "host":
            return _evolve(cfg, U0, case["steps"]).cpu()
        if case["kind"] == "routines":
            # V, F and G are the work arrays of a driver: only the state is the step's result
            return [_evolve(cfg, U0, 1), None, None, None]
        return _evolve(cfg, U0, case["steps"])


def _hash(z):
    """SplitMix64 in two's complement (the noise of the Kelvin-Helmholtz model)."""
    s = lambda v: v - (1 << 64) if v >> 63 else v  # noqa: E731
    r = lambda a, k: (a >> k) & ((1 << (64 - k)) - 1)  # noqa: E731
    z = z + s(0x9E3779B97F4A7C15)
    z = (z ^ r(z, 30)) * s(0xBF58476D1CE4E5B9)
    z = (z ^ r(z, 27)) * s(0x94D049BB133111EB)
    return z ^ r(z, 31)


def _model(cfg, m: ModelSpec):
    x, y, _ = _axes(cfg)
    if m.kind == 0:
        return _conserved(cfg, cfg.gamma ** 2, (-torch.sin(y + m.phase_y), torch.sin(x + m.phase_x), 0.0), cfg.gamma,
                          (-m.amp * torch.sin(y + m.phase_y), m.amp * torch.sin(2 * (x + m.phase_x)), 0.0))
    c = torch.arange(cfg.ix * cfg.jx, device="cuda").reshape(cfg.jx, cfg.ix)
    h = _hash(_hash(torch.tensor(m.seed, device="cuda")) ^ c)
    noise = ((h >> 11) & ((1 << 53) - 1)).double() * 2.0 ** -52 - 1
    return _conserved(cfg, 1.0, (m.amp * torch.tanh(y), m.pert * torch.exp(-y * y) * noise, 0.0), 0.5, (m.bx0, 0.0, 0.0))


def _signs(mask, U):
    return torch.tensor([-1.0 if (mask >> v) & 1 else 1.0 for v in range(9)], dtype=U.dtype, device=U.device).reshape(
        (9,) + (1,) * (U.dim() - 1))


def _fill(U, cfg):
    """Ghost cells, x sides first."""
    for a in range(cfg.nd):
        d = cfg.nd - a
        n = U.shape[d]
        first, last = U.narrow(d, 1, 1), U.narrow(d, n - 2, 1)
        if cfg.bc_kind[2 * a] == 0:
            lo, hi = last, first
        else:
            lo, hi = _signs(cfg.bc_flip[2 * a], U) * first, _signs(cfg.bc_flip[2 * a + 1], U) * last
        U = torch.cat([lo, U.narrow(d, 1, n - 2), hi], d)
    return U


def _primitive(U, gamma):
    v = U[0:3] / U[RO]
    p = (gamma - 1) * (U[EN] - 0.5 * ((v * U[0:3]).sum(0) + (U[5:8] ** 2).sum(0)))
    return torch.cat([v, p[None], U[4:9]])


def _inner(U, keep=None):
    """U without its ghost layers along every grid axis but `keep`."""
    for d in range(1, U.dim()):
        if d != keep:
            U = U.narrow(d, 1, U.shape[d] - 2)
    return U


def _speeds(U, cfg):
    """Largest |v| + fast speed of the interior."""
    w = _primitive(_inner(U), cfg.gamma)
    g, B2, s = cfg.gamma * w[PR], (w[5:8] ** 2).sum(0), 0.0
    for a in range(cfg.nd):
        D = (g + B2) ** 2 - 4 * g * w[BX + a] ** 2
        s = max(s, float((w[VX + a].abs() + torch.sqrt((g + B2 + torch.sqrt(D.clamp(min=0))) / (2 * w[RO]))).max()))
    return s


def _states(w, d, cfg, a):
    """States on both sides of the n - 1 faces along array axis d (grid axis a)."""
    n = w.shape[d]
    wm, w0, wp = (w.narrow(d, k, n - 2) for k in range(3))
    gA, gB = w0 - wm, wp - w0
    slope = torch.where(gB.abs() < gA.abs(), gB, gA)
    if cfg.limiter == "minmod":
        slope = 0.5 * slope
    else:
        gC = 0.25 * (wp - wm)
        one = torch.ones_like(gA)
        same = (torch.copysign(one, gA) * torch.copysign(one, gC)).detach()
        slope = torch.where(gC.abs() < slope.abs(), same * gC, slope)
    slope = torch.where(torch.signbit(gA) == torch.signbit(gB), slope, torch.zeros_like(slope))
    up, lo = w0 + slope, w0 - slope
    if cfg.bc_kind[2 * a] == 0:
        first, last = up.narrow(d, n - 3, 1), lo.narrow(d, 0, 1)
    else:
        first = _signs(cfg.bc_flip[2 * a], w) * lo.narrow(d, 0, 1)
        last = _signs(cfg.bc_flip[2 * a + 1], w) * up.narrow(d, n - 3, 1)
    return torch.cat([first, up], d), torch.cat([lo, last], d)


def _hlld(L, R, a, ch, gamma):
    """HLLD flux with the HLLC-G fallback and the GLM fluxes, normal along grid axis a; every
    quotient and root of a branch that is not taken is given a harmless operand."""
    n, t, u = a, (a + 1) % 3, (a + 2) % 3
    sgn = lambda x: torch.copysign(torch.ones_like(x), x).detach()  # noqa: E731

    def side(S):
        v, B, ro, p = S[0:3], S[5:8], S[RO], S[PR]
        B2, vB = (B * B).sum(0), (v * B).sum(0)
        pt = p + 0.5 * B2
        E = 0.5 * (ro * (v * v).sum(0) + B2) + p / (gamma - 1)
        U = [ro, ro * v[n], ro * v[t], ro * v[u], E, B[t], B[u]]
        F = [ro * v[n], ro * v[n] ** 2 + pt - B[n] ** 2, ro * v[n] * v[t] - B[n] * B[t], ro * v[n] * v[u] - B[n] * B[u],
             (E + pt) * v[n] - vB * B[n], v[n] * B[t] - B[n] * v[t], v[n] * B[u] - B[n] * v[u]]
        g = gamma * p
        c2 = (g + B2 + torch.sqrt(((g + B2) ** 2 - 4 * g * B[n] ** 2).clamp(min=0))) / (2 * ro)
        return U, F, vB, pt, c2

    UL, FL, vBL, ptL, cL = side(L)
    UR, FR, vBR, ptR, cR = side(R)
    cf = torch.sqrt(torch.where(cR > cL, cR, cL))
    vL, vR = L[n], R[n]
    aL = torch.where(vR < vL, vR, vL) - cf
    aR = torch.where(vR > vL, vR, vL) + cf
    isL = aL >= 0
    isR = ~isL & (aR <= 0)
    mid = ~(isL | isR)
    safe = lambda x, m: torch.where(m, x, torch.ones_like(x))  # noqa: E731
    f = 1 / (aR - aL)
    H = [f * (aR * p - aL * q - r + s) for p, q, r, s in zip(UR, UL, FR, FL)]
    Bn = f * (aR * R[BX + n] - aL * L[BX + n])
    hro = safe(H[0], mid)
    aM, at, au = H[1] / hro, H[2] / hro, H[3] / hro
    pt = ptL + L[RO] * (aL - vL) * (aM - vL)
    dL, dR = safe(aL - aM, mid), safe(aR - aM, mid)
    rL, rR = safe(L[RO] * (aL - vL) / dL, mid), safe(R[RO] * (aR - vR) / dR, mid)
    qL, qR = torch.sqrt(rL), torch.sqrt(rR)
    AL, AR = Bn.abs() / qL, Bn.abs() / qR
    isG = mid & ((aL >= aM - 1.001 * AL) | (aM + 1.001 * AR >= aR))
    star = mid & ~isG

    def energy(U, S, al, pS, vB, d, vt, vu, Bt, Bu):
        return ((al - S[n]) * U[4] - pS * S[n] + pt * aM + Bn * (vB - aM * Bn - vt * Bt - vu * Bu)) / d

    def jump(U, F, al, X):
        return [al * (x - q) + s for x, q, s in zip(X, U, F)]

    # HLLC-G
    eL = energy(UL, L, aL, ptL, vBL, dL, at, au, H[5], H[6])
    eR = energy(UR, R, aR, ptR, vBR, dR, at, au, H[5], H[6])
    gL = jump(UL, FL, aL, [rL, rL * aM, rL * at, rL * au, eL])
    gR = jump(UR, FR, aR, [rR, rR * aM, rR * at, rR * au, eR])
    left = ~torch.signbit(aM)
    fG = [torch.where(left, p, q) for p, q in zip(gL, gR)]
    fG += [f * (aR * FL[k] - aL * FR[k] + aL * aR * (UR[k] - UL[k])) for k in (5, 6)]

    # outer and central star states
    def outer(S, U, al, ro, d, vB, pS):
        k = 1 / safe(S[RO] * (al - S[n]) * (al - aM) - Bn * Bn, star)
        b = k * (S[RO] * (al - S[n]) ** 2 - Bn * Bn)
        Bt, Bu = S[BX + t] * b, S[BX + u] * b
        vt, vu = (S[q] - k * Bn * S[BX + q] * (aM - S[n]) for q in (t, u))
        return [ro, ro * aM, ro * vt, ro * vu, energy(U, S, al, pS, vB, safe(d, star), vt, vu, Bt, Bu), Bt, Bu], vt, vu

    XL, vtL, vuL = outer(L, UL, aL, rL, dL, vBL, ptL)
    XR, vtR, vuR = outer(R, UR, aR, rR, dR, vBR, ptR)
    isLs = star & (aM - AL >= 0)
    isRs = star & ~isLs & (aM + AR <= 0)
    s = sgn(Bn)
    k = 1 / (qL + qR)
    vt = k * (qL * vtL + qR * vtR + (XR[5] - XL[5]) * s)
    vu = k * (qL * vuL + qR * vuR + (XR[6] - XL[6]) * s)
    Bt = k * (qL * XR[5] + qR * XL[5] + qL * qR * (vtR - vtL) * s)
    Bu = k * (qL * XR[6] + qR * XL[6] + qL * qR * (vuR - vuL) * s)

    def central(X, q, ro, vt1, vu1, sg, a1, al, U, F):
        e = X[4] - sg * q * (vt1 * X[5] + vu1 * X[6] - vt * Bt - vu * Bu) * s
        Y = [ro, ro * aM, ro * vt, ro * vu, e, Bt, Bu]
        return [a1 * y - (a1 - al) * x - al * v + w for y, x, v, w in zip(Y, X, U, F)]

    cLs = central(XL, qL, rL, vtL, vuL, 1.0, aM - AL, aL, UL, FL)
    cRs = central(XR, qR, rR, vtR, vuR, -1.0, aM + AR, aR, UR, FR)
    sL, sR = jump(UL, FL, aL, XL), jump(UR, FR, aR, XR)
    out = [None] * 9
    for j, slot in enumerate((RO, MX + n, MX + t, MX + u, EN, BX + t, BX + u)):
        x = torch.where(aM >= 0, cLs[j], cRs[j])
        for where, val in ((isRs, sR), (isLs, sL), (isG, fG), (isR, FR), (isL, FL)):
            x = torch.where(where, val[j], x)
        out[slot] = x
    out[BX + n] = 0.5 * ((L[PS] + R[PS]) - ch * (R[BX + n] - L[BX + n]))
    out[PS] = 0.5 * (ch * ch * (L[BX + n] + R[BX + n]) - ch * (R[PS] - L[PS]))
    return torch.stack(out)


def _resistive(F, w, a, cfg):
    """Resistive parts of the fluxes along grid axis a (energy and the two tangential field components)."""
    nd = cfg.nd
    ax = _axes(cfg)
    pos = [None if x is None else x for x in ax]
    pos[a] = pos[a] + 0.5 * cfg.dx
    if cfg.eta == "recon2d":
        eta = 1e-3 + (1000.0 - 60.0) / 60000.0 / torch.cosh(torch.clamp(torch.sqrt(pos[0] ** 2 + pos[1] ** 2), max=25.0)) ** 2
    else:
        eta = 1e-3 + torch.exp(-(pos[0] ** 2 + pos[2] ** 2) / 4) / 60.0
    eta = torch.broadcast_to(eta, w.shape[1:])
    cut = lambda x, off: _cut(x, off, a, nd)  # noqa: E731
    eta = cut(eta, {}) / cfg.dx
    B = lambda c, **off: cut(w[BX + c], off)  # noqa: E731
    key = "xyz"

    def diff(c, b):  # dB_c/db at the face, times dx
        if b >= nd:
            return 0.0
        if b == a:
            return B(c, **{key[a]: 1}) - B(c)
        up = B(c, **{key[b]: 1}) + B(c, **{key[a]: 1, key[b]: 1})
        dn = B(c, **{key[b]: -1}) + B(c, **{key[a]: 1, key[b]: -1})
        return 0.25 * (up - dn)

    t, u = (a + 1) % 3, (a + 2) % 3
    Jt = eta * (diff(a, u) - diff(u, a))
    Ju = eta * (diff(t, a) - diff(a, t))
    mean = lambda c: B(c) + B(c, **{key[a]: 1})  # noqa: E731
    F = list(F)
    F[EN] = F[EN] + 0.5 * (Jt * mean(u) - Ju * mean(t))
    F[BX + t] = F[BX + t] - Ju
    F[BX + u] = F[BX + u] + Jt
    return torch.stack(F)


def _cut(x, off, a, nd):
    """x at the cells below the faces along grid axis a (interior along the others), moved by `off` cells."""
    for b in range(nd):
        d = x.dim() - 1 - b
        o = off.get("xyz"[b], 0)
        n = x.shape[d]
        x = x.narrow(d, o, n - 1) if b == a else x.narrow(d, 1 + o, n - 2)
    return x


def _divergence(U, cfg, dt, ch):
    w = _primitive(U, cfg.gamma)
    D = 0.0
    for a, h in zip(range(cfg.nd), (cfg.dx, cfg.dy, cfg.dz)):
        d = cfg.nd - a
        L, R = _states(_inner(w, keep=d), d, cfg, a)
        F = _hlld(L, R, a, ch, cfg.gamma)
        if cfg.eta != "none":
            F = _resistive(F, w, a, cfg)
        n = F.shape[d]
        D = D + dt / h * (F.narrow(d, 0, n - 1) - F.narrow(d, 1, n - 1))
    return torch.nn.functional.pad(D, (1, 1) * cfg.nd)


def _evolve(cfg, U, steps):
    U = _fill(U, cfg)
    hmin = min((cfg.dx, cfg.dy, cfg.dz)[: cfg.nd])
    for _ in range(steps):
        with torch.no_grad():
            ch = _speeds(U, cfg)
        dt = cfg.cfl * hmin / ch
        if cfg.eta == "recon2d":
            dt = min(dt, 0.5 * cfg.cfl * 60.0 * cfg.dx ** 2)
        elif cfg.eta == "harris_xz":
            dt = min(dt, 0.5 * cfg.cfl / (1e-3 + 1 / 60.0) * cfg.dx ** 2)
        damp = torch.ones(9, dtype=U.dtype, device=U.device)
        damp[PS] = math.exp(-0.5 * dt * ch / 0.2)
        damp = damp.reshape((9,) + (1,) * cfg.nd)
        U = damp * U
        U1 = _fill(U + _divergence(U, cfg, dt, ch), cfg)
        U = damp * _fill(0.5 * (U + U1 + _divergence(U1, cfg, dt, ch)), cfg)
    return U
