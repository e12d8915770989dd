"""The work that users of this framework have it do, as cases that can be timed and checked.

Each case goes through the public entry points of the package (heat_run, heat_stage, burgers_run,
burgers_run_fixed, heatk_run, weno7_run, Ensemble) with the state, plan and workspaces that a
program keeps between calls. `exact` states the same schemes in plain FP64 torch."""
import math
import random

import torch

from multigpu_advectiondiffusion_gb300 import _native as N
from multigpu_advectiondiffusion_gb300 import solvers as S


def listed():
    return [
        # The smallest call: one O4 SSP-RK3 stage of a small grid, issued by a program that drives
        # its own time loop (ragged rows; launch and call cost count as much as the kernel).
        {"name": "heat stage 65x61x57 f32", "kind": "heat_stage", "scheme": "reference", "nx": 65, "ny": 61, "nz": 57,
         "dtype": "f32", "stage": 2},
        # 2D heat, the plain benchmark problem: 512^2, 5-point, forward Euler, 1000 steps.
        {"name": "heat2d 512 f32", "kind": "heat_run", "scheme": "dirichlet", "nx": 512, "ny": 512, "nz": 1,
         "dtype": "f32", "steps": 1000},
        # 3D heat, the headline problem: 256^3, 7-point, forward Euler (a part of its 2000 steps).
        {"name": "heat3d 256 f32", "kind": "heat_run", "scheme": "dirichlet", "nx": 256, "ny": 256, "nz": 256,
         "dtype": "f32", "steps": 200},
        # The reference program's own run: O4 + SSP-RK3 in FP64 on its 201 x 199 x 200 nodes.
        {"name": "heat3d reference f64", "kind": "heat_run", "scheme": "reference", "nx": 201, "ny": 199, "nz": 200,
         "dtype": "f64", "steps": 10},
        # 3D Burgers, the benchmark problem: periodic 256^3 WENO5-Z, global Lax-Friedrichs, dt from
        # max|u|, the default weight division.
        {"name": "burgers3d 256 z f32", "kind": "burgers_run", "scheme": "periodic", "nx": 256, "ny": 256, "nz": 256,
         "dtype": "f32", "weno": "z", "lf": "global", "div": "f64", "steps": 4},
        # The reference program's scheme in its own precision: frozen layers, local Lax-Friedrichs,
        # WENO5-Z, viscous term, fixed dt, FP64, odd sizes.
        {"name": "burgers3d reference f64", "kind": "burgers_run", "scheme": "reference", "nx": 121, "ny": 101, "nz": 97,
         "dtype": "f64", "weno": "z", "lf": "local", "div": "f32", "steps": 2},
        # A small ragged problem in FP32, WENO5-JS: a user's first try, where launches count.
        {"name": "burgers3d small js f32", "kind": "burgers_run", "scheme": "reference", "nx": 61, "ny": 53, "nz": 47,
         "dtype": "f32", "weno": "js", "lf": "local", "div": "f32", "steps": 8},
        # 2D Burgers as the reference's 2D program has it (WENO5-JS, local, inviscid), FP32.
        {"name": "burgers2d 1000x900 f32", "kind": "burgers_run", "scheme": "reference_2d", "nx": 1000, "ny": 900,
         "nz": 1, "dtype": "f32", "weno": "js", "lf": "local", "div": "f32", "steps": 8},
        # Gradient of a Burgers run with respect to its initial state (forward and backward).
        {"name": "burgers gradient 128 f32", "kind": "burgers_grad", "nx": 128, "ny": 128, "nz": 128, "dtype": "f32",
         "weno": "z", "steps": 10},
        # Gradient of a heat run with respect to its diffusivity field (forward and backward).
        {"name": "heatk gradient 192 f32", "kind": "heatk_grad", "nx": 192, "ny": 192, "nz": 192, "dtype": "f32",
         "steps": 40},
        # Many problems of uneven size in one graph: heat and Burgers members together.
        {"name": "ensemble 16+8 f32", "kind": "ensemble", "heat": 16, "burgers": 8, "mix": 4, "dtype": "f32",
         "steps": 20},
        # The seventh-order prototype scheme, LSRK(5,4), FP32.
        {"name": "weno7 160 f32", "kind": "weno7_run", "nx": 160, "ny": 160, "nz": 160, "dtype": "f32", "steps": 3},
    ]


# A drawn case costs no more than the largest listed one: flop counts of its passes (see _flops).
_CAP = 6.0e10


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _steps(rng, per_step, hi):
    most = max(1, min(hi, int(_CAP / max(per_step, 1.0))))
    return _log_int(rng, 1, most)


def draw(rng):
    kind = rng.choice(["heat_stage", "heat_run", "heat_run", "heat2d", "burgers_run", "burgers_run", "burgers2d",
                       "burgers_grad", "heatk_grad", "ensemble", "weno7_run"])
    if kind in ("heat_stage", "heat_run", "heat2d"):
        f64 = rng.random() < 0.35
        c = {"kind": "heat_stage" if kind == "heat_stage" else "heat_run",
             "scheme": rng.choice(["dirichlet", "reference"]), "dtype": "f64" if f64 else "f32"}
        if kind == "heat2d":
            n = _log_int(rng, 64, 2048)
            c.update(nx=n, ny=max(32, int(n * rng.uniform(0.6, 1.1))), nz=1)
        else:
            n = _log_int(rng, 24, 256)
            c.update(nx=n, ny=max(16, int(n * rng.uniform(0.7, 1.0))), nz=max(12, int(n * rng.uniform(0.5, 1.0))))
        if c["scheme"] == "dirichlet":  # that constructor takes one node count
            c.update(ny=c["nx"], nz=1 if c["nz"] == 1 else c["nx"])
        if kind == "heat_stage":
            c["stage"] = 1 if c["scheme"] == "dirichlet" else rng.choice([1, 2, 3])
        else:
            c["steps"] = _steps(rng, _flops({**c, "steps": 1}) * (20 if f64 else 1), 1000)
        return c
    if kind == "burgers_run":
        f64 = rng.random() < 0.35
        per = rng.random() < 0.5
        n = _log_int(rng, 24, 128 if f64 else 256)
        c = {"kind": kind, "scheme": "periodic" if per else "reference", "nx": n, "ny": n, "nz": n,
             "dtype": "f64" if f64 else "f32", "weno": rng.choice(["z", "z", "js"]),
             "lf": rng.choice(["global", "local"]) if per else "local",
             "div": rng.choice(["f32", "f64", "f64", "fast"])}
        if not per:
            c.update(ny=max(16, int(n * rng.uniform(0.7, 1.0))), nz=max(14, int(n * rng.uniform(0.6, 1.0))))
        c["steps"] = _steps(rng, _flops({**c, "steps": 1}) * (20 if f64 else 1), 12)
        return c
    if kind == "burgers2d":
        n = _log_int(rng, 100, 2000)
        c = {"kind": "burgers_run", "scheme": "reference_2d", "nx": n, "ny": max(64, int(n * rng.uniform(0.6, 1.1))),
             "nz": 1, "dtype": "f32", "weno": "js", "lf": "local", "div": "f32"}
        c["steps"] = _steps(rng, _flops({**c, "steps": 1}), 16)
        return c
    if kind == "burgers_grad":
        n = _log_int(rng, 24, 128)
        c = {"kind": kind, "nx": n, "ny": n, "nz": n, "dtype": "f32", "weno": "z"}
        c["steps"] = _steps(rng, _flops({**c, "steps": 1}), 12)
        return c
    if kind == "heatk_grad":
        n = _log_int(rng, 32, 192)
        c = {"kind": kind, "nx": n, "ny": n, "nz": n, "dtype": "f32"}
        c["steps"] = _steps(rng, _flops({**c, "steps": 1}), 60)
        return c
    if kind == "ensemble":
        c = {"kind": kind, "heat": rng.randint(2, 20), "burgers": rng.randint(1, 8), "mix": rng.randint(0, 10 ** 6),
             "dtype": "f32"}
        c["steps"] = _steps(rng, _flops({**c, "steps": 1}), 24)
        return c
    n = _log_int(rng, 24, 160)
    twod = rng.random() < 0.25
    c = {"kind": "weno7_run", "nx": 4 * n if twod else n, "ny": 3 * n if twod else n, "nz": 1 if twod else n,
         "dtype": "f32"}
    c["steps"] = _steps(rng, _flops({**c, "steps": 1}), 6)
    return c


# ------------------------------------------------------------------------------- the problems
def _dtype(c):
    return torch.float32 if c["dtype"] == "f32" else torch.float64


def _heat_cfg(c):
    if c["scheme"] == "dirichlet":
        return S.HeatConfig.dirichlet_o2(2 if c["nz"] == 1 else 3, c["nx"])
    if c["nz"] == 1:
        return S.HeatConfig.reference_2d(1.0, 10.0, 10.0, c["nx"], c["ny"])
    return S.HeatConfig.reference_3d(1.0, 10.0, 10.0, 10.0, c["nx"], c["ny"], c["nz"])


def _burgers_cfg(c):
    if c["scheme"] == "periodic":
        return S.BurgersConfig.periodic(c["nx"], weno=c["weno"], lf=c["lf"], div=c["div"])
    if c["scheme"] == "reference_2d":
        return S.BurgersConfig.reference_2d(2.0, 2.0, c["nx"], c["ny"])
    cfg = S.BurgersConfig.reference(2.0, 2.0, 2.0, c["nx"], c["ny"], c["nz"])
    cfg.weno = N.ADV_WENO5_Z if c["weno"] == "z" else N.ADV_WENO5_JS
    cfg.div = {"f32": N.ADV_DIV_F32, "f64": N.ADV_DIV_F64, "fast": N.ADV_DIV_FAST}[c["div"]]
    return cfg


def _members(c):
    """Sizes and diffusivities of an ensemble's members (the benchmark's choices of them)."""
    r = random.Random(c["mix"])
    heat = [(r.choice([64, 96, 128, 160, 192]), 10.0 ** r.uniform(-1, 1)) for _ in range(c["heat"])]
    return heat, [r.choice([96, 112, 128, 144, 160]) for _ in range(c["burgers"])]


def _grid(n, dev):
    return torch.linspace(0.0, 1.0, n, dtype=torch.float64, device=dev)


def _blobs(nx, ny, nz, gen, dtype):
    """Eight Gaussian blobs on the unit square or cube, zero on the boundary nodes."""
    dev = torch.device("cuda")
    x, y, z = _grid(nx, dev), _grid(ny, dev), _grid(nz, dev)
    u = torch.zeros(nz, ny, nx, dtype=torch.float64, device=dev)
    p = torch.rand(8, 4, generator=gen, dtype=torch.float64, device=dev).cpu()
    for cx, cy, cz, w in p.tolist():
        s = 1.0 / (2.0 * (0.02 + 0.06 * w) ** 2)
        g = [torch.exp(-s * (v - (0.2 + 0.6 * m)) ** 2) for v, m in ((x, cx), (y, cy), (z, cz))]
        gz = g[2] if nz > 1 else torch.ones_like(g[2])
        u += gz[:, None, None] * g[1][None, :, None] * g[0][None, None, :]
    u[:, 0, :] = u[:, -1, :] = 0
    u[:, :, 0] = u[:, :, -1] = 0
    if nz > 1:
        u[0] = u[-1] = 0
    return u.to(dtype).contiguous()


def _fourier(nx, ny, nz, gen, dtype):
    """0.5 plus sixteen random Fourier modes of the periodic box."""
    dev = torch.device("cuda")
    x, y, z = (torch.arange(n, dtype=torch.float64, device=dev) / n for n in (nx, ny, nz))
    u = torch.full((nz, ny, nx), 0.5, dtype=torch.float64, device=dev)
    k = torch.randint(-4, 5, (16, 3), generator=gen, device=dev).cpu().tolist()
    a = torch.rand(16, 2, generator=gen, dtype=torch.float64, device=dev).cpu().tolist()
    for (kx, ky, kz), (amp, ph) in zip(k, a):
        fx, fy, fz = (torch.exp(2j * math.pi * m * v) for m, v in ((kx, x), (ky, y), (kz if nz > 1 else 0, z)))
        m = fz[:, None, None] * (fy[None, :, None] * fx[None, None, :] * complex(math.cos(6.28 * ph), math.sin(6.28 * ph)))
        u += 0.1 * amp * m.real
    return u.to(dtype).contiguous()


def _initial(c, gen):
    dt = _dtype(c)
    if c["kind"] in ("heat_run", "heat_stage"):
        return _blobs(c["nx"], c["ny"], c["nz"], gen, dt)
    if c["kind"] == "weno7_run" or c["kind"] == "burgers_run" and c["scheme"] != "periodic":
        # smooth bumps of either sign, |u| of about 1 as the reference's fixed time step assumes
        return (0.6 * _blobs(c["nx"], c["ny"], c["nz"], gen, torch.float64)
                - 0.4 * _fourier(c["nx"], c["ny"], c["nz"], gen, torch.float64)).to(dt).contiguous()
    return _fourier(c["nx"], c["ny"], c["nz"], gen, dt)


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    kind = c["kind"]
    if kind == "heat_stage":
        cfg, u = _heat_cfg(c), _initial(c, gen)
        un = _initial(c, gen) if c["stage"] > 1 else u
        return {"c": c, "cfg": cfg, "u": u, "un": un, "out": torch.empty_like(u)}
    if kind == "heat_run":
        cfg, u0 = _heat_cfg(c), _initial(c, gen)
        return {"c": c, "cfg": cfg, "u0": u0, "u": torch.empty_like(u0), "ws": S.heat_workspace(cfg, u0)}
    if kind == "burgers_run":
        cfg, u0 = _burgers_cfg(c), _initial(c, gen)
        return {"c": c, "cfg": cfg, "u0": u0, "u": torch.empty_like(u0), "ws": S.burgers_workspace(cfg, u0)}
    if kind == "weno7_run":
        cfg = S.Weno7Config(c["nx"], c["ny"], c["nz"], *_weno7_h(c))
        u0 = _initial(c, gen)
        return {"c": c, "cfg": cfg, "u0": u0, "u": torch.empty_like(u0), "ws": S.weno7_workspace(cfg, u0)}
    if kind == "burgers_grad":
        cfg = S.BurgersConfig.periodic(c["nx"], weno=c["weno"], lf="local", div="f64")
        u0, target = _initial(c, gen), _initial(c, gen)
        return {"c": c, "cfg": cfg, "u0": u0.requires_grad_(True), "target": target, "dt": _grad_dt(c)}
    if kind == "heatk_grad":
        u0, target = (_blobs(c["nx"], c["ny"], c["nz"], gen, _dtype(c)) for _ in range(2))
        k = _diffusivity(c, gen)
        return {"c": c, "cfg": S.HeatKConfig.cube(c["nx"], 0.125, _K_MAX), "u0": u0.requires_grad_(True),
                "k": k.requires_grad_(True), "target": target}
    heat, burgers = _members(c)
    hu0 = [_blobs(n, n, n, gen, torch.float32) for n, _ in heat]
    bu0 = [_fourier(n, n, n, gen, torch.float32) for n in burgers]
    hu, bu = [torch.empty_like(u) for u in hu0], [torch.empty_like(u) for u in bu0]
    ens = S.Ensemble(heat=[(S.HeatConfig.dirichlet_o2(3, n, k=k, r=0.125), u) for (n, k), u in zip(heat, hu)],
                     burgers=[(S.BurgersConfig.periodic(n, weno="z", div="f64"), u, 1e9, 0.4, N.ADV_DT_MAXU, c["steps"])
                              for n, u in zip(burgers, bu)])
    return {"c": c, "ens": ens, "u0": hu0 + bu0, "u": hu + bu}


_K_MAX = 4.0


def _diffusivity(c, gen):
    """Log-normal diffusivity, smooth over the box, at most _K_MAX."""
    f = _fourier(c["nx"], c["ny"], c["nz"], gen, torch.float64) - 0.5
    return torch.exp(2.0 * f).clamp_(max=_K_MAX).to(_dtype(c)).contiguous()


def _weno7_h(c):
    return tuple(2.0 / max(n - 1, 1) for n in (c["nx"], c["ny"], c["nz"]))


def _grad_dt(c):
    return 0.2 * (2.0 / c["nx"])


_FAR = 1e9  # an end time that the step limit comes before


def run(state):
    c, kind = state["c"], state["c"]["kind"]
    if kind == "heat_stage":
        S.heat_stage(state["cfg"], c["stage"], state["u"], state["un"], state["out"])
        return state["out"]
    if kind == "heat_run":
        state["u"].copy_(state["u0"])
        return S.heat_run(state["cfg"], state["u"], c["steps"], workspace=state["ws"])
    if kind == "burgers_run":
        state["u"].copy_(state["u0"])
        rule = N.ADV_DT_MAXU if c["scheme"] == "periodic" else N.ADV_DT_FIXED
        t, steps = S.burgers_run(state["cfg"], state["u"], _FAR, 0.4, rule, max_steps=c["steps"], workspace=state["ws"])
        return {"u": state["u"], "t": t, "steps": steps}
    if kind == "weno7_run":
        state["u"].copy_(state["u0"])
        t, steps = S.weno7_run(state["cfg"], state["u"], _FAR, 0.4, max_steps=c["steps"], workspace=state["ws"])
        return {"u": state["u"], "t": t, "steps": steps}
    if kind == "burgers_grad":
        u = S.burgers_run_fixed(state["cfg"], state["u0"], state["dt"], c["steps"])
        (g,) = torch.autograd.grad(0.5 * (u - state["target"]).square().sum(), (state["u0"],))
        return {"u": u.detach(), "grad": g}
    if kind == "heatk_grad":
        u = S.heatk_run(state["cfg"], state["k"], state["u0"], c["steps"])
        gk, gu = torch.autograd.grad(0.5 * (u - state["target"]).square().sum(), (state["k"], state["u0"]))
        return {"u": u.detach(), "grad_k": gk, "grad_u": gu}
    for u, u0 in zip(state["u"], state["u0"]):
        u.copy_(u0)
    state["ens"].run(c["steps"])
    return state["u"]


# ------------------------------------------------------------------------------------- the work
def _flops(c):
    """Floating-point operations of one pass (a fused multiply-add counts as two)."""
    kind = c["kind"]
    if kind == "ensemble":
        heat, burgers = _members(c)
        return c["steps"] * (16.0 * sum(n ** 3 for n, _ in heat) + 3 * 380.0 * sum(n ** 3 for n in burgers))
    n = float(c["nx"] * c["ny"] * c["nz"])
    axes = 2 if c["nz"] == 1 else 3
    if kind in ("heat_run", "heat_stage"):
        stage = (5.0 * axes + 1) if c["scheme"] == "dirichlet" else (9.0 * axes + 5)
        stages = 1 if kind == "heat_stage" else c["steps"] * (1 if c["scheme"] == "dirichlet" else 3)
        return stages * stage * n
    if kind == "burgers_run":
        return c["steps"] * 3 * n * (120.0 * axes + 20)
    if kind == "weno7_run":
        return c["steps"] * 5 * n * (260.0 * axes + 20)
    if kind == "burgers_grad":
        return c["steps"] * 3 * n * 1140.0
    return c["steps"] * n * 90.0  # heatk_grad: the step and its adjoint


def work(case):
    c = case
    size = 4 if c["dtype"] == "f32" else 8
    if c["kind"] == "ensemble":
        heat, burgers = _members(c)
        return {"bytes": 2.0 * size * (sum(n ** 3 for n, _ in heat) + sum(n ** 3 for n in burgers)), "flops": _flops(c)}
    arrays = {"heat_stage": 3 if c.get("stage", 1) > 1 else 2, "heat_run": 2, "burgers_run": 2, "weno7_run": 2,
              "burgers_grad": 4, "heatk_grad": 6}[c["kind"]]
    return {"bytes": float(arrays * size * c["nx"] * c["ny"] * c["nz"]), "flops": _flops(c)}


# ------------------------------------------------------------------- the same schemes in FP64
def _sh(u, axis, d):
    """u at index i + d along an axis (wrapped; the frozen schemes read no wrapped value)."""
    return torch.roll(u, -d, dims=axis)


def _inner(u, layers):
    """True on the nodes at least `layers` away from every face (a 2D grid has no z faces)."""
    m = torch.zeros(u.shape, dtype=torch.bool, device=u.device)
    F = layers
    z = slice(None) if u.shape[0] == 1 else slice(F, u.shape[0] - F)
    m[z, F:u.shape[1] - F, F:u.shape[2] - F] = True
    return m


def _axes(u):
    return ((2, "x"), (1, "y")) if u.shape[0] == 1 else ((2, "x"), (1, "y"), (0, "z"))


def _heat_L(cfg, u):
    L = torch.zeros_like(u)
    for ax, name in _axes(u):
        k = getattr(cfg, "k" + name)
        if cfg.order == 2:
            L += k * (_sh(u, ax, 1) - 2 * u + _sh(u, ax, -1))
        else:
            L += k * (-_sh(u, ax, 2) + 16 * _sh(u, ax, 1) - 30 * u + 16 * _sh(u, ax, -1) - _sh(u, ax, -2))
    return L


def _heat_stage64(cfg, stage, u, un, inner, outer):
    v = u + cfg.dt * _heat_L(cfg, u)
    r = un + cfg.dt * _heat_L(cfg, u) if stage == 1 else 0.75 * un + 0.25 * v if stage == 2 else (un + 2 * v) / 3
    r = torch.where(inner, r, u)
    return torch.where(outer, torch.zeros_like(r), r) if cfg.zero_boundary else r


def _heat64(cfg, u, steps):
    inner, outer = _inner(u, cfg.frozen), ~_inner(u, 1)
    for _ in range(steps):
        if cfg.time == N.ADV_EULER:
            u = _heat_stage64(cfg, 1, u, u, inner, outer)
        else:
            a = _heat_stage64(cfg, 1, u, u, inner, outer)
            b = _heat_stage64(cfg, 2, a, u, inner, outer)
            u = _heat_stage64(cfg, 3, b, u, inner, outer)
    return u


def _weno5(a, b, c, d, e, z):
    eps = 1e-6
    b0 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    b1 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b2 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    if z:
        tau = (b0 - b2).abs()
        w0, w1, w2 = 0.1 * (1 + tau / (b0 + eps)), 0.6 * (1 + tau / (b1 + eps)), 0.3 * (1 + tau / (b2 + eps))
    else:
        w0, w1, w2 = 0.1 / (b0 + eps) ** 2, 0.6 / (b1 + eps) ** 2, 0.3 / (b2 + eps) ** 2
    num = w0 * (2 * a - 7 * b + 11 * c) + w1 * (-b + 5 * c + 2 * d) + w2 * (2 * c + 5 * d - e)
    return num / (6 * (w0 + w1 + w2))


def _burgers_L(cfg, u, alpha):
    L = torch.zeros_like(u)
    a = u.abs() if alpha is None else alpha
    f = 0.5 * u * u
    fp, fm = 0.5 * (f + a * u), 0.5 * (f - a * u)
    z = cfg.weno == N.ADV_WENO5_Z
    for ax, name in _axes(u):
        F = _weno5(*(_sh(fp, ax, j) for j in (-2, -1, 0, 1, 2)), z) + _weno5(*(_sh(fm, ax, j) for j in (3, 2, 1, 0, -1)), z)
        h = getattr(cfg, "d" + name)
        L -= (F - _sh(F, ax, -1)) / h
        if cfg.C:
            L += cfg.C / (12 * h * h) * (-_sh(u, ax, 2) + 16 * _sh(u, ax, 1) - 30 * u + 16 * _sh(u, ax, -1) - _sh(u, ax, -2))
    return L


def _burgers_stage64(cfg, stage, u, un, dt, inner):
    alpha = u.abs().max() if cfg.lf == N.ADV_LF_GLOBAL else None
    v = u + dt * _burgers_L(cfg, u, alpha)
    r = v if stage == 1 else 0.75 * un + 0.25 * v if stage == 2 else (un + 2 * v) / 3
    return r if inner is None else torch.where(inner, r, u)


def _burgers_step64(cfg, u, dt, inner):
    a = _burgers_stage64(cfg, 1, u, u, dt, inner)
    b = _burgers_stage64(cfg, 2, a, u, dt, inner)
    return _burgers_stage64(cfg, 3, b, u, dt, inner)


def _burgers64(cfg, u, steps, max_rule):
    inner = None if cfg.bc == N.ADV_BC_PERIODIC else _inner(u, 3)
    t = 0.0
    for _ in range(steps):
        dt = 0.4 * cfg.dx / float(u.abs().max()) if max_rule else _fixed_dt(cfg, u.shape[0] == 1)
        u = _burgers_step64(cfg, u, dt, inner)
        t += dt
    return u, t


def _fixed_dt(cfg, twod):
    iz = 0.0 if twod else 1 / cfg.dz / cfg.dz
    dt = 0.9 / (2 * cfg.C * (1 / cfg.dx / cfg.dx + 1 / cfg.dy / cfg.dy + iz)) if cfg.C else math.inf
    return min(0.4 * cfg.dx, dt)


# WENO7: the indicators beta_k as the prototype's integer quadratic forms over a candidate's four
# cells (coefficients of x0^2, x0 x1, x0 x2, x0 x3, x1^2, x1 x2, x1 x3, x2^2, x2 x3, x3^2).
_W7_BETA = [
    (6649, -47214, 56694, -22778, 85641, -210282, 86214, 134241, -114894, 25729),
    (3169, -19374, 19014, -5978, 33441, -70602, 23094, 41001, -30414, 6649),
    (6649, -30414, 23094, -5978, 41001, -70602, 19014, 33441, -19374, 3169),
    (25729, -114894, 86214, -22778, 134241, -210282, 56694, 85641, -47214, 6649),
]
_W7_CAND = [(-3, 13, -23, 25), (1, -5, 13, 3), (-1, 7, 7, -1), (3, 13, -5, 1), (25, -23, 13, -3)]
_W7_LIN = (1 / 35, 12 / 35, 18 / 35, 4 / 35)


def _weno7_part(f, plus):
    num = den = 0.0
    for k in range(4):
        x = f[k:k + 4]
        i, beta = 0, 0.0
        for p in range(4):
            for q in range(p, 4):
                beta = beta + _W7_BETA[k][i] * (x[p] * x[q])
                i += 1
        w = (_W7_LIN[k] if plus else _W7_LIN[3 - k]) / (1e-6 + beta) ** 2
        cand = _W7_CAND[k] if plus else _W7_CAND[k + 1]
        num = num + w * sum(m * v for m, v in zip(cand, x)) / 12
        den = den + w
    return num / den


def _weno7_R(cfg, u):
    R = torch.zeros_like(u)
    f, au = 0.5 * u * u, u.abs() * u
    fp, fm = 0.5 * (f + au), 0.5 * (f - au)
    for ax, name in _axes(u):
        n = u.shape[ax]
        at = [(torch.arange(n, device=u.device) + d).clamp(0, n - 1) for d in range(-3, 5)]
        H = _weno7_part([fp.index_select(ax, at[j]) for j in range(7)], True)
        H += _weno7_part([fm.index_select(ax, at[j]) for j in range(1, 8)], False)
        left = torch.roll(H, 1, dims=ax)
        left.select(ax, 0).zero_()
        R += (H - left) / getattr(cfg, "d" + name)
    return R


_LSRK_A = (0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0,
           -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0)
_LSRK_B = (1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0, 1720146321549.0 / 2090206949498.0,
           3134564353537.0 / 4481467310338.0, 2277821191437.0 / 14882151754819.0)


def _weno7_64(cfg, u, steps):
    t, r = 0.0, torch.zeros_like(u)
    for _ in range(steps):
        dt = 0.4 * cfg.dx / float(u.abs().max())
        for a, b in zip(_LSRK_A, _LSRK_B):
            r = a * r + dt * _weno7_R(cfg, u)
            u = u - b * r
        t += dt
    return u, t


def _heatk_step64(cfg, k, u, inner):
    r = u
    for ax, name in _axes(u):
        kp, km = 0.5 * (k + _sh(k, ax, 1)), 0.5 * (k + _sh(k, ax, -1))
        r = r + getattr(cfg, "c" + name) * (kp * (_sh(u, ax, 1) - u) - km * (u - _sh(u, ax, -1)))
    return torch.where(inner, r, torch.zeros_like(u) if cfg.zero_boundary else u)


def exact(case, seed):
    c = case
    s = prepare(c, seed)
    kind = c["kind"]
    with torch.no_grad():
        if kind == "heat_stage":
            u, un = s["u"].double(), s["un"].double()
            return _heat_stage64(s["cfg"], c["stage"], u, un, _inner(u, s["cfg"].frozen), ~_inner(u, 1))
        if kind == "heat_run":
            return _heat64(s["cfg"], s["u0"].double(), c["steps"])
        if kind == "burgers_run":
            u, t = _burgers64(s["cfg"], s["u0"].double(), c["steps"], c["scheme"] == "periodic")
            return {"u": u, "t": t, "steps": None}
        if kind == "weno7_run":
            u, t = _weno7_64(s["cfg"], s["u0"].double(), c["steps"])
            return {"u": u, "t": t, "steps": None}
        if kind == "ensemble":
            heat, burgers = _members(c)
            got = [_heat64(S.HeatConfig.dirichlet_o2(3, n, k=k, r=0.125), u.double(), c["steps"])
                   for (n, k), u in zip(heat, s["u0"])]
            return got + [_burgers64(S.BurgersConfig.periodic(n, weno="z", div="f64"), u.double(), c["steps"], True)[0]
                          for n, u in zip(burgers, s["u0"][len(heat):])]
    # the gradients: torch's own differentiation of the FP64 steps, one step at a time
    u = s["u0"].detach().double()
    if kind == "burgers_grad":
        if c["nx"] * c["ny"] * c["nz"] > 160 ** 3:
            return None
        step, k = (lambda v, _: _burgers_step64(s["cfg"], v, s["dt"], None)), None
    else:
        inner, k = _inner(u, 1), s["k"].detach().double()
        step = lambda v, kk: _heatk_step64(s["cfg"], kk, v, inner)  # noqa: E731
    states = [u]
    with torch.no_grad():
        for _ in range(c["steps"]):
            states.append(step(states[-1], k))
    lam = states[-1] - s["target"].double()
    gk = torch.zeros_like(u)
    for v in reversed(states[:-1]):
        v = v.requires_grad_(True)
        kk = None if k is None else k.clone().requires_grad_(True)
        w = step(v, kk)
        if k is None:
            (lam,) = torch.autograd.grad(w, (v,), lam)
        else:
            lam, g = torch.autograd.grad(w, (v, kk), lam)
            gk += g
        v.requires_grad_(False)
    return {"u": states[-1], "grad": lam} if k is None else {"u": states[-1], "grad_k": gk, "grad_u": lam}
