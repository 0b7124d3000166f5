"""The work this framework does for its users, as timed cases.

Every kind of case is one thing that a program does with the package: advance
a flow (the differentiable step, the interactive step with its V-cycles, the
converging step with and without the learned warm start, a batch of channels),
solve a pressure equation, differentiate a rollout, train the warm start, or
use the predictor and the post-step fields on their own.  ``listed`` has the
sizes of the package's configurations and benchmark, with ragged and odd ones
beside them; ``draw`` spreads the same kinds over their ranges.

``exact`` restates each case in float64 with plain torch on the same inputs.
The projection's discrete operators are those of the reference solver: edge
ghosts, outlet pressure row pinned at 0, the inlet at x = 0 and walls in y.
"""
import functools
import math

import torch
import torch.nn.functional as F

import aerojax_gb300 as aj
from aerojax_gb300 import adjoint, ensemble, nn

DEV = "cuda"
H = 1.0 / 64.0           # grid spacing of the package's configurations
NET_FACTOR = 8           # fine cells per cell of the warm start's grid


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one differentiable step on the small validation channel: the
        # shortest call a time loop makes, where launches count
        {"name": "pure_512x96", "kind": "pure", "nx": 512, "ny": 96, "cycles": 3},
        # the interactive solver's step with its default five V-cycles
        {"name": "gui_mac_2048x512", "kind": "gui", "nx": 2048, "ny": 512, "cycles": 5},
        # a short run from an impulsive start, pressure converged every step
        # from the previous one
        {"name": "converge_mac_2048x512", "kind": "converge", "nx": 2048, "ny": 512, "steps": 4},
        # the same run with the learned warm start: the package's headline
        {"name": "learned_mac_2048x512", "kind": "learned", "nx": 2048, "ny": 512, "steps": 4},
        # the largest configuration: dynamic LES and hyperviscosity
        {"name": "cylinders_4096x2048", "kind": "cylinders", "nx": 4096, "ny": 2048, "steps": 2},
        # a parameter study: channels of uneven sizes stepped as one batch
        {"name": "ensemble_16", "kind": "ensemble", "count": 16, "draw_seed": 0},
        # a pressure solve by itself on a ragged grid, both solvers
        {"name": "solve_1440x352", "kind": "solve", "nx": 1440, "ny": 352},
        {"name": "vcycle_mac_1008x368", "kind": "vcycle", "nx": 1008, "ny": 368, "cycles": 5},
        # the gradient of a loss of a rollout's end (inverse design)
        {"name": "gradient_512x128", "kind": "gradient", "nx": 512, "ny": 128, "steps": 8},
        # the gradient of one training batch of the warm start
        {"name": "train_16x256x64", "kind": "train", "batch": 16, "h": 256, "w": 64},
        # the predictor with its eddy viscosity alone, on an odd grid
        {"name": "predictor_1021x509", "kind": "predictor", "nx": 1021, "ny": 509, "mac": True,
         "weno": True},
        # what a viewer asks for after a step: dye, vorticity, divergence, speed
        {"name": "post_4096x2048", "kind": "post", "nx": 4096, "ny": 2048, "mac": False},
    ]


def _log(rng, lo, hi, multiple=1):
    """A size between lo and hi, uniform in its logarithm."""
    return max(1, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / multiple)) * multiple


def _grid(rng, lo, hi, multiple, aspect=(2.0, 6.0)):
    """An elongated grid of nx in [lo, hi]; both sizes multiples of ``multiple``."""
    nx = _log(rng, lo, hi, multiple)
    ny = max(2 * multiple, round(nx / rng.uniform(*aspect) / multiple) * multiple)
    return nx, ny


def _converging(rng, lo, hi, aspect=(2.0, 6.0)):
    """A grid that the converging solver takes: halved while both sizes are
    even, it ends on at most 1024 cells."""
    while True:
        nx, ny = _grid(rng, lo, hi, 64, aspect)
        n, m = nx, ny
        while n % 2 == 0 and m % 2 == 0 and n * m > 64:
            n, m = n // 2, m // 2
        if n * m <= 1024:
            return nx, ny


def draw(rng):
    kind = rng.choice(["pure", "gui", "converge", "learned", "cylinders", "ensemble", "solve",
                       "vcycle", "gradient", "train", "predictor", "post"])
    c = {"kind": kind}
    if kind == "pure":
        c["nx"], c["ny"] = _grid(rng, 128, 2048, 16)
        c["cycles"] = rng.choice([1, 2, 3, 5])
    elif kind == "gui":
        c["nx"], c["ny"] = _grid(rng, 256, 3072, 16)
        c["cycles"] = rng.choice([3, 5])
    elif kind in ("converge", "learned"):
        c["nx"], c["ny"] = _converging(rng, 256, 2048)
        c["steps"] = rng.randint(2, 4)
    elif kind == "cylinders":
        c["nx"], c["ny"] = _converging(rng, 512, 4096, (2.0, 3.0))
        c["steps"] = 2
    elif kind == "ensemble":
        c["count"], c["draw_seed"] = rng.randint(4, 21), rng.randint(1, 1 << 20)
    elif kind == "solve":
        c["nx"], c["ny"] = _converging(rng, 192, 4096)
    elif kind == "vcycle":
        c["nx"], c["ny"] = _grid(rng, 128, 4096, 16)
        c["cycles"] = rng.choice([1, 3, 5])
    elif kind == "gradient":
        c["nx"], c["ny"] = _grid(rng, 128, 1024, 16)
        c["steps"] = rng.randint(2, 10)
    elif kind == "train":
        c["batch"], c["h"], c["w"] = _log(rng, 2, 16), _log(rng, 64, 256, 8), _log(rng, 32, 64, 8)
    else:
        c["nx"], c["ny"] = _grid(rng, 67, 4096, 1)
        c["mac"] = rng.random() < 0.5
        if kind == "predictor":
            c["weno"] = rng.random() < 0.5
    return c


# ------------------------------------------------------------------ inputs
def _coords(nx, ny):
    x = torch.arange(nx, device=DEV, dtype=torch.float64)[:, None] * (nx * H / (nx - 1))
    y = torch.arange(ny, device=DEV, dtype=torch.float64)[None, :] * (ny * H / (ny - 1))
    return x, y


@functools.lru_cache(maxsize=None)
def _obstacle(kind, nx, ny):
    """(mask, sdf) of the obstacle: a NACA 0012 section at 10 degrees, three
    cylinders on a triangle, or one cylinder.  A program has one geometry for
    many flows, so one per grid is kept."""
    x, y = _coords(nx, ny)
    lx, ly = nx * H, ny * H
    if kind == "naca":
        chord, a = lx / 8, math.radians(10.0)
        px, py = x - 0.2 * lx, y - 0.5 * ly
        xr = px * math.cos(a) - py * math.sin(a)
        yr = px * math.sin(a) + py * math.cos(a)
        s = (xr / chord).clamp(0.0, 1.0)
        t = 0.6 * chord * (0.2969 * s.sqrt() - 0.126 * s - 0.3516 * s ** 2 + 0.2843 * s ** 3
                           - 0.1015 * s ** 4)
        out = (xr - s * chord).abs()
        sdf = torch.where(out > 0, (out ** 2 + yr ** 2).sqrt(), yr.abs() - t)
    elif kind == "cylinders":
        d, gap = ly / 32, ly / 12.8
        sdf = None
        for dx, dy in ((-1 / math.sqrt(3.0), 0.0), (0.5 / math.sqrt(3.0), 0.5),
                       (0.5 / math.sqrt(3.0), -0.5)):
            one = ((x - 0.2 * lx - dx * gap) ** 2 + (y - 0.5 * ly - dy * gap) ** 2).sqrt() - d / 2
            sdf = one if sdf is None else torch.minimum(sdf, one)
    else:
        sdf = ((x - 0.19 * lx) ** 2 + (y - 0.5 * ly) ** 2).sqrt() - ly / 12
    mask = 1.0 - torch.sigmoid(-sdf / (0.05 * H))
    return mask.float().contiguous(), sdf.float().contiguous()


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _flow(nx, ny, seed, mac=False):
    """A free stream with large eddies on it and the start-up noise of the
    package's configurations; on the faces for a MAC grid."""
    g = _gen(seed)
    r = torch.rand(12, generator=g, device=DEV, dtype=torch.float64)

    def field(n, m, a, b):
        x = torch.arange(n, device=DEV, dtype=torch.float64)[:, None] / n
        y = torch.arange(m, device=DEV, dtype=torch.float64)[None, :] / m
        f = (0.05 * torch.sin(2 * math.pi * (3 * x + r[a])) * torch.sin(math.pi * (2 * y + r[a + 1]))
             + 0.03 * torch.sin(2 * math.pi * (7 * x + r[a + 2])) * torch.cos(math.pi * (5 * y + r[b])))
        return f + 1e-3 * torch.randn(n, m, generator=g, device=DEV, dtype=torch.float64)

    u = 1.0 + field(nx + 1 if mac else nx, ny, 0, 3)
    v = field(nx, ny + 1 if mac else ny, 4, 7)
    return u.float().contiguous(), v.float().contiguous()


def _rhs(nx, ny, seed):
    """A pressure equation's right-hand side: eddies, and a grid-scale part."""
    g = _gen(seed)
    x, y = _coords(nx, ny)
    b = torch.randn(nx, ny, generator=g, device=DEV, dtype=torch.float64)
    r = torch.rand(24, generator=g, device=DEV, dtype=torch.float64)
    for k in range(8):
        wide = (0.02 + 0.05 * r[3 * k]) * ny * H
        d2 = (x - r[3 * k + 1] * nx * H) ** 2 + (y - r[3 * k + 2] * ny * H) ** 2
        b = b + (40.0 if k % 2 else -40.0) * torch.exp(-d2 / wide ** 2)
    return b.float().contiguous()


def _net_params(seed):
    return nn.init_params(seed % 1000)


def _train_data(case, seed):
    g = _gen(seed)
    n, h, w = case["batch"], case["h"], case["w"]
    x3 = torch.randn(n, h, w, 3, generator=g, device=DEV)
    x3 = F.avg_pool2d(x3.permute(0, 3, 1, 2), 3, 1, 1).permute(0, 2, 3, 1).contiguous()
    return x3, 0.5 * x3[..., 0] + 0.1 * torch.randn(n, h, w, generator=g, device=DEV)


# ------------------------------------------------------------------ state
def _config(case):
    """The StepConfig of a stepping case, as the package's configurations set it."""
    k, nx, ny = case["kind"], case["nx"], case["ny"]
    base = dict(nx=nx, ny=ny, dx=H, dy=H, U_inf=1.0, cfl_dt=True, dt=0.5 * H, cfl_target=0.5,
                dt_min=1e-6, dt_max=1.0, variant="gui", use_les=True, brinkman_eta=1e-4)
    if k == "cylinders":
        return aj.StepConfig(nu=ny * H / 32 / 3000.0, grid_type="collocated",
                             les_model="dynamic_smagorinsky", nu_hyper_ratio=0.01,
                             mg_mode="converge", max_cycles=60, has_sdf=True, warm_start=True,
                             **base)
    mac = dict(nu=nx * H / 8 / 1000.0, grid_type="mac", les_model="smagorinsky",
               smagorinsky_constant=0.17)
    if k == "gui":
        return aj.StepConfig(mg_mode="parity", v_cycles=case["cycles"], **mac, **base)
    return aj.StepConfig(mg_mode="converge", max_cycles=60, warm_start=True,
                         nn_factor=NET_FACTOR if k == "learned" else 0, **mac, **base)


def _steps_of(case):
    return case.get("steps", 1)


def _specs(case):
    return ensemble.draw_instances(case["count"], seed=case["draw_seed"])


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case}
    if k == "pure":
        s["mask"], s["sdf"] = _obstacle("cylinder", case["nx"], case["ny"])
        u, v = _flow(case["nx"], case["ny"], seed)
        s["state"] = aj.SimState(u=u, v=v, p=torch.zeros_like(u), u_prev=u, v_prev=v, c=None,
                                 dt=0.4 * H, iteration=0)
    elif k in ("gui", "converge", "learned", "cylinders"):
        cfg = _config(case)
        mac = cfg.grid_type == "mac"
        s["mask"], sdf = _obstacle("naca" if mac else "cylinders", case["nx"], case["ny"])
        s["plan"] = aj.Plan(cfg, DEV)
        s["plan"].prepare(s["mask"], sdf if cfg.has_sdf else None)
        u, v = _flow(case["nx"], case["ny"], seed, mac)
        s["first"] = (u, v, torch.zeros_like(s["mask"]))
        s["bufs"] = [tuple(torch.empty_like(t) for t in s["first"]) for _ in range(2)]
        if k == "learned":
            s["net"] = nn.WarmStartNet.load(nn.WEIGHTS, device=DEV)
    elif k == "ensemble":
        s["ens"] = ensemble.Ensemble(_specs(case), device=DEV, seed=seed % 100000)
    elif k in ("solve", "vcycle"):
        s["mask"], _ = _obstacle("cylinder", case["nx"], case["ny"])
        s["rhs"] = _rhs(case["nx"], case["ny"], seed)
    elif k == "gradient":
        s["mask"], s["sdf"] = _obstacle("cylinder", case["nx"], case["ny"])
        u, v = _flow(case["nx"], case["ny"], seed)
        s["state"] = aj.SimState(u=u, v=v, p=torch.zeros_like(u), u_prev=u, v_prev=v, c=None,
                                 dt=0.3 * H, iteration=0)
        s["params"] = {"dx": H, "dy": H, "nu": 2e-3, "U_inf": 1.0, "sdf": s["sdf"]}
        s["g"] = tuple(_flow(case["nx"], case["ny"], seed + 7919))
    elif k == "train":
        s["net"] = nn.WarmStartNet(device=DEV, params=_net_params(seed))
        s["x3"], s["target"] = _train_data(case, seed)
    elif k == "predictor":
        s["mask"], sdf = _obstacle("cylinder", case["nx"], case["ny"])
        s["sdf"] = None if case["mac"] else sdf
        s["u"], s["v"] = _flow(case["nx"], case["ny"], seed, case["mac"])
        s["uc"], s["vc"] = _flow(case["nx"], case["ny"], seed + 1)
    else:
        s["u"], s["v"] = _flow(case["nx"], case["ny"], seed, case["mac"])
        s["c"] = torch.rand(case["nx"], case["ny"], generator=_gen(seed + 1), device=DEV)
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "pure":
        st = aj.step_pure(s["state"], s["mask"], s["sdf"], H, H, 1.5e-3, 1.0,
                          v_cycles=case["cycles"], brinkman_eta=1e-4)
        return {"u": st.u, "v": st.v, "p": st.p}
    if k in ("gui", "converge", "learned", "cylinders"):
        u, v, p = s["first"]
        warm = s["plan"].cfg.warm_start
        for i in range(_steps_of(case)):
            out = s["bufs"][i % 2]
            if k == "learned":
                u, v, p = nn.run_step_nn(s["plan"], s["net"], u, v, s["mask"], p, out=out)
            else:
                u, v, p = aj.run_step(s["plan"], u, v, s["mask"], p_guess=p if warm else None,
                                      out=out)
        return {"u": u, "v": v, "p": p}
    if k == "ensemble":
        s["ens"].step()
        return [s["ens"].state(i) for i in range(case["count"])]
    if k == "solve":
        return aj.poisson_multigrid_converge(s["rhs"], s["mask"], H, H, rtol=1e-6)[0]
    if k == "vcycle":
        return aj.poisson_multigrid_mac(s["rhs"], s["mask"], H, H, v_cycles=case["cycles"])
    if k == "gradient":
        end, hist = adjoint.differentiable_rollout(s["state"], s["mask"], s["params"],
                                                   case["steps"])
        g = adjoint.rollout_vjp(s["state"], s["mask"], s["params"], case["steps"], *s["g"],
                                history=hist)
        return {"end": [end.u, end.v, end.p], "g": [g["u"], g["v"], g["sdf"]], "nu": g["nu"],
                "U_inf": g["U_inf"]}
    if k == "train":
        n, h, w, net = case["batch"], case["h"], case["w"], s["net"]
        net.expand(s["x3"], n, h, w)
        y = net.forward(None, n, h, w)
        loss, dy = net.loss(y, s["target"], n, h, w)
        return {"y": y, "loss": loss, "grad": net.backward(dy, n, h, w)}
    if k == "predictor":
        sgs = aj.constant_smagorinsky(s["uc"], s["vc"], H, H, H, C_s=0.17)
        adv = "weno5" if case["weno"] else "upwind"
        if case["mac"]:
            us, vs = aj.rk_step_unified_mac(s["u"], s["v"], 0.3 * H, 1e-3, H, H, s["mask"],
                                            nu_sgs=sgs, brinkman_eta=1e-4, advection=adv)
        else:
            us, vs = aj.rk_step_unified(s["u"], s["v"], 0.3 * H, 1e-3, H, H, s["mask"], s["sdf"],
                                        nu_sgs=sgs, brinkman_eta=1e-4, advection=adv)
        return {"u": us, "v": vs, "sgs": sgs}
    return list(aj.post_step(s["u"], s["v"], s["c"], 0.3 * H, H, H, 1e-3,
                             grid_type="mac" if case["mac"] else "collocated"))


# ------------------------------------------------------------------ work
def _conv_flops(n, h, w):
    """Multiply-adds of one pass of the warm start's network, as two flops."""
    halved = [0, 0, 1, 1, 2, 2, 3, 3, 2, 1, 0, 0]
    return sum(18.0 * n * (h >> l) * (w >> l) * ci * co for (ci, co, _), l in zip(nn.LAYERS, halved))


def work(case):
    """Inputs read once and outputs written once, in 32 bits; the arithmetic
    that the method asks for, per cell: about 80 for each Runge-Kutta stage
    (350 with WENO5), 60 for a V-cycle's sweeps and transfers, three of which
    bring a warm-started solve to its tolerance."""
    k = case["kind"]
    if k == "train":
        n, h, w = case["batch"], case["h"], case["w"]
        p = sum(9 * ci * co + co for ci, co, _ in nn.LAYERS)
        return {"bytes": 4.0 * (n * h * w * (3 + 1 + 16) + 2 * p), "flops": 3 * _conv_flops(n, h, w)}
    if k == "ensemble":
        cells = sum(s.nx * s.ny for s in _specs(case))
        return {"bytes": 28.0 * cells, "flops": (3 * 350 + 3 * 60) * cells}
    cells = case["nx"] * case["ny"]
    if k == "pure":
        return {"bytes": 28.0 * cells, "flops": (240 + 60 * case["cycles"]) * cells}
    if k == "gui":
        return {"bytes": 24.0 * cells, "flops": (280 + 60 * case["cycles"]) * cells}
    if k in ("converge", "learned", "cylinders"):
        net = _conv_flops(1, case["nx"] // NET_FACTOR, case["ny"] // NET_FACTOR) if k == "learned" else 0
        les = 300 if k == "cylinders" else 40
        one = {"bytes": (32.0 if k == "cylinders" else 28.0) * cells,
               "flops": (240 + les + 3 * 60) * cells + net}
        return {m: _steps_of(case) * one[m] for m in one}
    if k == "solve":
        return {"bytes": 8.0 * cells, "flops": 5 * 60.0 * cells}
    if k == "vcycle":
        return {"bytes": 12.0 * cells, "flops": 60.0 * case["cycles"] * cells}
    if k == "gradient":
        # forward: the state in, the history out; reverse: the history in
        return {"bytes": 4.0 * cells * (4 * case["steps"] + 12), "flops": 3 * 300.0 * case["steps"] * cells}
    if k == "predictor":
        return {"bytes": 4.0 * cells * 9, "flops": 3 * (350 if case["weno"] else 80.0) * cells}
    return {"bytes": 28.0 * cells, "flops": 60.0 * cells}


# ------------------------------------------------------------------ float64
def _edge(f, a, b):
    """Edge padding by a rows and b columns on each side."""
    n, m = f.shape
    i = torch.arange(-a, n + a, device=f.device).clamp(0, n - 1)
    j = torch.arange(-b, m + b, device=f.device).clamp(0, m - 1)
    return f[i][:, j]


def _lap(f):
    p = _edge(f, 1, 1)
    return ((p[2:, 1:-1] + p[:-2, 1:-1] - 2 * f) + (p[1:-1, 2:] + p[1:-1, :-2] - 2 * f)) / H ** 2


def _central(f, axis):
    """Central differences, one-sided in the first and last row (or column)."""
    p = _edge(f, 1 - axis, axis)
    n = f.shape[axis]
    d = p.narrow(axis, 2, n) - p.narrow(axis, 0, n)
    w = torch.full((n,), 0.5 / H, device=f.device, dtype=f.dtype)
    w[0] = w[-1] = 1.0 / H
    return d * (w[:, None] if axis == 0 else w[None, :])


def _upwind(f, vel, axis):
    p = _edge(f, 1 - axis, axis)
    n = f.shape[axis]
    back, fwd = f - p.narrow(axis, 0, n), p.narrow(axis, 2, n) - f
    return vel * torch.where(vel > 0, back, fwd) / H


def _weno(f, vel, axis):
    """Jiang and Shu's fifth-order upwind derivative, edge ghosts."""
    p = _edge(f, 3 * (1 - axis), 3 * axis)
    n = f.shape[axis]
    d = p.diff(dim=axis) / H

    def side(idx):
        a, b, c, e, g = (d.narrow(axis, q, n) for q in idx)
        w1 = 0.1 / (1e-6 + 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2) ** 2
        w2 = 0.6 / (1e-6 + 13 / 12 * (b - 2 * c + e) ** 2 + 0.25 * (b - e) ** 2) ** 2
        w3 = 0.3 / (1e-6 + 13 / 12 * (c - 2 * e + g) ** 2 + 0.25 * (3 * c - 4 * e + g) ** 2) ** 2
        return (w1 * (a / 3 - 7 / 6 * b + 11 / 6 * c) + w2 * (-b / 6 + 5 / 6 * c + e / 3)
                + w3 * (c / 3 + 5 / 6 * e - g / 6)) / (w1 + w2 + w3)

    return vel * torch.where(vel > 0, side((0, 1, 2, 3, 4)), side((5, 4, 3, 2, 1)))


def _channel_bc(u, v, U=1.0):
    """Inlet, outflow copy, slip walls (u) and no flow through them (v)."""
    u = torch.cat([torch.zeros_like(u[:1]) + U, u[1:-1], u[-2:-1]])
    v = torch.cat([torch.zeros_like(v[:1]), v[1:-1], v[-2:-1]])
    u = torch.cat([u[:, 1:2], u[:, 1:-1], u[:, -2:-1]], 1)
    z = torch.zeros_like(v[:, :1])
    return u, torch.cat([z, v[:, 1:-1], z], 1)


def _rk3(u, v, dt, rhs, den_u, den_v):
    k1 = rhs(u, v)
    k2 = rhs((u + dt * k1[0]) / den_u, (v + dt * k1[1]) / den_v)
    k3 = rhs((u + 0.25 * dt * k2[0]) / den_u, (v + 0.25 * dt * k2[1]) / den_v)
    return (u + 2 / 3 * dt * k3[0]) / den_u, (v + 2 / 3 * dt * k3[1]) / den_v


def _predict(u, v, dt, nu, mask, chi, eta, sgs=0.0, hyper=0.0, nu_hyper=None, weno=False, U=1.0):
    """Collocated predictor; nu + sgs is the viscosity."""
    adv = _weno if weno else _upwind

    def rhs(a, b):
        la, lb = _lap(a), _lap(b)
        ra = -adv(a, a, 0) - adv(a, b, 1) + (nu + sgs) * la
        rb = -adv(b, a, 0) - adv(b, b, 1) + (nu + sgs) * lb
        if hyper > 0:
            ra, rb = ra - nu_hyper * _lap(la), rb - nu_hyper * _lap(lb)
        return ra, rb

    den = 1 + dt * chi / eta
    u, v = _rk3(u, v, dt, rhs, den, den)
    solid = mask <= 0.5
    return _channel_bc(u.masked_fill(solid, 0.0), v.masked_fill(solid, 0.0), U)


def _to_faces(c, axis):
    p = _edge(c, 1 - axis, axis)
    n = c.shape[axis]
    return 0.5 * (p.narrow(axis, 0, n + 1) + p.narrow(axis, 1, n + 1))


def _to_cells(f, axis):
    n = f.shape[axis] - 1
    return 0.5 * (f.narrow(axis, 0, n) + f.narrow(axis, 1, n))


def _predict_mac(u, v, dt, nu, mask32, eta, sgs, weno=False):
    """Staggered predictor.  The walls' test, chi on the face below one half,
    is a decision on 32-bit data and is taken on it."""
    mask = mask32.double()
    mu, mv = _to_faces(mask, 0), _to_faces(mask, 1)
    cu, cv = _to_faces(1.0 - mask, 0), _to_faces(1.0 - mask, 1)
    nu_u, nu_v = nu + _to_faces(sgs, 0), nu + _to_faces(sgs, 1)

    def blend(f, axis):
        p = _edge(f, 1 - axis, axis)
        n = f.shape[axis]
        w = 0.5 * (1 + torch.tanh(f / 0.05))
        return f * (w * (f - p.narrow(axis, 0, n)) + (1 - w) * (p.narrow(axis, 2, n) - f)) / H

    def rhs(a, b):
        wu, wv = _channel_bc(a, b)
        vu = _to_faces(_to_cells(wv, 1), 0)
        uv = _to_faces(_to_cells(wu, 0), 1)
        if weno:
            au = _weno(wu, wu, 0) + _weno(wu, vu, 1)
            av = _weno(wv, uv, 0) + _weno(wv, wv, 1)
        else:
            au = blend(wu, 0) + vu * _central(wu, 1)
            av = uv * _central(wv, 0) + blend(wv, 1)
        return -au * mu + nu_u * _lap(a), -av * mv + nu_v * _lap(b)

    u, v = _rk3(u, v, dt, rhs, 1 + dt * cu / eta, 1 + dt * cv / eta)
    chi32 = 1.0 - mask32
    u = u.masked_fill(_to_faces(chi32, 0) >= 0.5, 0.0)
    v = v.masked_fill(_to_faces(chi32, 1) >= 0.5, 0.0)
    return _channel_bc(u, v)


def _strain(u, v):
    """Periodic velocity gradients' strain rate, as the eddy viscosities use it."""
    def g(f, a):
        return (f.roll(-1, a) - f.roll(1, a)) / (2 * H)
    xx, yy, xy = g(u, 0), g(v, 1), 0.5 * (g(u, 1) + g(v, 0))
    return (2 * (xx ** 2 + yy ** 2 + 2 * xy ** 2) + 1e-10).sqrt(), xx, yy, xy


def _smagorinsky(u, v, cs):
    return (cs * H) ** 2 * _strain(u, v)[0]


def _dynamic(u, v):
    def box(f):
        return sum(f.roll(i, 0).roll(j, 1) for i in range(-2, 3) for j in range(-2, 3)) / 25

    def near(f):
        out = torch.zeros_like(f)
        n, m = f.shape
        out[1:-1, 1:-1] = sum(f[i:n - 2 + i, j:m - 2 + j] for i in range(3) for j in range(3)) / 9
        return out

    s, xx, yy, xy = _strain(u, v)
    a, b = box(u), box(v)
    st, txx, tyy, txy = _strain(a, b)
    l11, l12, l22 = a * a - box(u * u), a * b - box(u * v), b * b - box(v * v)
    m11, m12, m22 = 4 * st * txx - box(s * xx), 4 * st * txy - box(s * xy), 4 * st * tyy - box(s * yy)
    lm = near(l11 * m11 + l12 * m12 + l22 * m22)
    mm = near(m11 * m11 + m12 * m12 + m22 * m22)
    return (lm / (mm + 1e-8)).clamp(0.0, 0.2) * H * H * s


def _pin(b):
    return torch.cat([b[:-1], torch.zeros_like(b[-1:])])


def _solve(b):
    """The pressure equation's solution: cosine modes in y, and in x those of
    an edge ghost at the inlet and a value of 0 in the outlet row."""
    n, m = b.shape
    j = torch.arange(m, device=b.device, dtype=b.dtype)
    cy = torch.cos(math.pi * j[:, None] * (2 * j[None, :] + 1) / (2 * m)) * math.sqrt(2.0 / m)
    cy[0] = math.sqrt(1.0 / m)
    i = torch.arange(n - 1, device=b.device, dtype=b.dtype)
    th = (2 * i + 1) * math.pi / (2 * n - 1)
    cx = torch.cos(th[:, None] * (i[None, :] + 0.5)) * math.sqrt(4.0 / (2 * n - 1))
    lam = (-4 / H ** 2) * (torch.sin(th / 2)[:, None] ** 2
                           + torch.sin(math.pi * j / (2 * m))[None, :] ** 2)
    x = cx.T @ ((cx @ b[:-1] @ cy.T) / lam) @ cy
    return torch.cat([x, torch.zeros_like(b[-1:])])


def _vcycles(rhs, cycles, mask=None):
    """The reference's V-cycles from zero: two undamped Jacobi sweeps each way
    on every level, all levels at the finest spacing, ten sweeps on the
    coarsest; with a mask, the staggered grid's form."""
    b = _pin(rhs if mask is None else rhs * mask)
    n, m = b.shape
    depth = 1
    while n % 2 == 0 and m % 2 == 0 and depth < 4:
        n, m, depth = n // 2, m // 2, depth + 1

    def sweeps(p, r, k, count):
        for _ in range(count):
            e = _edge(p, 1, 1)
            p = ((e[2:, 1:-1] + e[:-2, 1:-1] + e[1:-1, 2:] + e[1:-1, :-2]) - H * H * r) / 4
            p = p if k is None else p * k
        return p

    def residual(p, r):
        a = _lap(p)
        return r - (a if mask is None else _pin(a))

    def halve(f):
        return 0.25 * (f[::2, ::2] + f[1::2, ::2] + f[::2, 1::2] + f[1::2, 1::2])

    def finer(c, axis):
        """Even points copied, odd ones the mean of their two; the last one 0."""
        k = c.shape[axis]
        mid = 0.5 * (c.narrow(axis, 0, k - 1) + c.narrow(axis, 1, k - 1))
        mid = torch.cat([mid, torch.zeros_like(c.narrow(axis, 0, 1))], axis)
        return torch.stack([c, mid], axis + 1).flatten(axis, axis + 1)

    def cycle(p, r, k, level):
        if level >= depth:
            return sweeps(p, r, k, 10)
        p = _pin(sweeps(p, r, k, 2))
        rc = halve(residual(p, r))
        kc = None if k is None else (halve(k) > 0.5).to(r.dtype)
        p = p + finer(finer(cycle(torch.zeros_like(rc), rc, kc, level + 1), 0), 1)
        return _pin(sweeps(p, r, k, 2))

    p = torch.zeros_like(b)
    for _ in range(cycles):
        p = cycle(p, b, mask, 0)
        if float((residual(p, b) ** 2).sum()) * H * H < 1e-12:
            break
    return p


def _divergence(u, v):
    d = torch.zeros_like(u)
    d[1:-1, 1:-1] = ((u[2:, 1:-1] - u[:-2, 1:-1]) + (v[1:-1, 2:] - v[1:-1, :-2])) / (2 * H)
    return d


def _pure(u, v, dt, nu, mask, sdf, eta, pressure, U=1.0, weno=False):
    us, vs = _predict(u, v, dt, nu, mask, torch.sigmoid(-sdf / (0.1 * H)), eta, weno=weno, U=U)
    p = pressure(_divergence(us, vs) * mask / dt)
    px, py = _central(p, 0), _central(p, 1)
    mx, my = _central(mask, 0), _central(mask, 1)
    g = (mx ** 2 + my ** 2).sqrt()
    nx, ny = mx / (g + 1e-8), my / (g + 1e-8)
    along = px * nx + py * ny
    wall = g > 0.1 / H
    px, py = torch.where(wall, px - along * nx, px), torch.where(wall, py - along * ny, py)
    px = torch.cat([torch.zeros_like(px[:1]), px[1:]])
    solid = mask <= 0.5
    un = (us - dt * px).masked_fill(solid, 0.0)
    vn = (vs - dt * py).masked_fill(solid, 0.0)
    un, vn = _channel_bc(un, vn, U)
    return un.masked_fill(solid, 0.0), vn.masked_fill(solid, 0.0), p


def _gui_bc(u, v):
    u[0, 1:-1], v[0] = 1.0, 0.0
    u[-1], v[-1] = u[-2], v[-2]
    u[:, 0] = u[:, -1] = 0.0
    v[:, 0] = v[:, -1] = 0.0
    return u, v


def _cfl(u, v, nu):
    top = (u.abs().max(), v.abs().max()) if u.shape != v.shape else ((u ** 2 + v ** 2).sqrt().max(),)
    return 0.5 * min(H / (max(map(float, top)) + 1e-12), 0.25 * H * H / (nu + 1e-12))


def _gui_mac(u, v, nu, mask32, pressure):
    dt = _cfl(u, v, nu)
    sgs = _smagorinsky(_to_cells(u, 0), _to_cells(v, 1), 0.17)
    us, vs = _predict_mac(u, v, dt, nu, mask32, 1e-4, sgs)
    p = pressure((us.diff(dim=0) + vs.diff(dim=1)) / H / dt)
    px, py = _edge(p, 1, 0).diff(dim=0) / H, _edge(p, 0, 1).diff(dim=1) / H
    px[0] = 0.0
    return (*_gui_bc(us - dt * px, vs - dt * py), p)


def _gui_cylinders(u, v, nu, mask, sdf):
    dt = _cfl(u, v, nu)
    sgs = _dynamic(u, v)
    # the interactive step hands the predictor nu + sgs as nu, and sgs again
    us, vs = _predict(u, v, dt, nu + sgs, mask, torch.sigmoid(-sdf / (0.1 * H)), 1e-4, sgs, 0.01,
                      (nu + sgs) * 0.01 * H * H)
    p = _solve(_pin(_divergence(us, vs) / dt))
    px, py = _central(p, 0), _central(p, 1)
    px[0] = 0.0
    un, vn = _gui_bc(us - dt * px, vs - dt * py)
    solid = mask <= 0.5
    return un.masked_fill(solid, 0.0), vn.masked_fill(solid, 0.0), p


def _exact_ensemble(case, seed):
    out = []
    for i, spec in enumerate(_specs(case)):
        cfg, mask, sdf, u, v = ensemble.instance_case(spec, DEV, seed % 100000 + i)
        u, v, mask, sdf = (t.double() for t in (u, v, mask, sdf))
        out.append(_pure(u, v, _cfl(u, v, cfg.nu), cfg.nu, mask, sdf, cfg.brinkman_eta,
                         lambda b: _solve(_pin(b)), weno=True))
    return out


def _exact_gradient(case, seed):
    mask, sdf32 = _obstacle("cylinder", case["nx"], case["ny"])
    u0, v0 = (t.double().requires_grad_() for t in _flow(case["nx"], case["ny"], seed))
    sdf = sdf32.double().requires_grad_()
    nu = torch.tensor(2e-3, device=DEV, dtype=torch.float64, requires_grad=True)
    U = torch.tensor(1.0, device=DEV, dtype=torch.float64, requires_grad=True)
    u, v = u0, v0
    for _ in range(case["steps"]):
        u, v, p = _pure(u, v, 0.3 * H, nu, mask.double(), sdf, 0.005, lambda b: _vcycles(b, 1), U)
    gu, gv = (t.double() for t in _flow(case["nx"], case["ny"], seed + 7919))
    g = torch.autograd.grad((u * gu).sum() + (v * gv).sum(), (u0, v0, sdf, nu, U))
    return {"end": [u.detach(), v.detach(), p.detach()], "g": list(g[:3]), "nu": float(g[3]),
            "U_inf": float(g[4])}


def _exact_train(case, seed):
    x3, target = _train_data(case, seed)
    flat = torch.as_tensor(_net_params(seed), device=DEV).double().requires_grad_()
    layers, o = [], 0
    for ci, co, relu in nn.LAYERS:
        w = flat[o:o + 9 * ci * co].view(3, 3, ci, co).permute(3, 2, 0, 1)
        o += 9 * ci * co
        layers.append((w, flat[o:o + co], relu))
        o += co

    def conv(x, k):
        w, b, relu = layers[k]
        x = F.conv2d(x, w, b, padding=1)
        return x.relu() if relu else x

    def up(x):
        return F.interpolate(x, scale_factor=2, mode="nearest")

    x = F.pad(x3.double(), (0, 13)).permute(0, 3, 1, 2)
    s0 = conv(conv(x, 0), 1)
    s1 = conv(conv(F.avg_pool2d(s0, 2), 2), 3)
    s2 = conv(conv(F.avg_pool2d(s1, 2), 4), 5)
    d = up(conv(conv(F.avg_pool2d(s2, 2), 6), 7)) + s2
    d = up(conv(d, 8)) + s1
    d = up(conv(d, 9)) + s0
    y = conv(conv(d, 10), 11).permute(0, 2, 3, 1)
    loss = ((y[..., 0] - target.double()) ** 2).mean()
    return {"y": y.detach().contiguous(), "loss": loss.detach()[None],
            "grad": torch.autograd.grad(loss, flat)[0]}


def _exact_post(case, seed):
    u, v = (t.double() for t in _flow(case["nx"], case["ny"], seed, case["mac"]))
    c = torch.rand(case["nx"], case["ny"], generator=_gen(seed + 1), device=DEV).double()

    def second(f, axis):
        p = _edge(f, 1 - axis, axis)
        n = f.shape[axis]
        return (p.narrow(axis, 2, n) + p.narrow(axis, 0, n) - 2 * f) / H ** 2

    def middle(f, axis):
        p = _edge(f, 1 - axis, axis)
        n = f.shape[axis]
        return (p.narrow(axis, 2, n) - p.narrow(axis, 0, n)) / (2 * H)

    if case["mac"]:
        uc, vc = _to_cells(u, 0), _to_cells(v, 1)
        # the reference pairs each component with its own direction here
        vort = middle(uc, 0) - middle(vc, 1)
        div = (u.diff(dim=0) + v.diff(dim=1)) / H
        rate = -uc * middle(c, 0) - vc * middle(c, 1) + 1e-3 * (second(c, 0) + second(c, 1))
    else:
        uc, vc = u, v
        vort = _central(v, 0) - _central(u, 1)
        div = _divergence(u, v)
        cy = (c.roll(-1, 1) - c.roll(1, 1)) / (2 * H)
        lap = second(c, 0) + (c.roll(1, 1) + c.roll(-1, 1) - 2 * c) / H ** 2
        rate = -u * _central(c, 0) - v * cy + 1e-3 * lap
    return [(c + 0.3 * H * rate).clamp(0.0, 1.0), vort, div, (uc ** 2 + vc ** 2).sqrt()]


def exact(case, seed):
    k = case["kind"]
    if k == "ensemble":
        return _exact_ensemble(case, seed)
    if k == "gradient":
        return _exact_gradient(case, seed)
    if k == "train":
        return _exact_train(case, seed)
    if k == "post":
        return _exact_post(case, seed)
    nx, ny = case["nx"], case["ny"]
    if k == "solve":
        return _solve(_pin(_rhs(nx, ny, seed).double()))
    if k == "vcycle":
        return _vcycles(_rhs(nx, ny, seed).double(), case["cycles"],
                        _obstacle("cylinder", nx, ny)[0].double())
    if k == "predictor":
        mask, sdf = _obstacle("cylinder", nx, ny)
        u, v = (t.double() for t in _flow(nx, ny, seed, case["mac"]))
        sgs = _smagorinsky(*(t.double() for t in _flow(nx, ny, seed + 1)), 0.17)
        if case["mac"]:
            u, v = _predict_mac(u, v, 0.3 * H, 1e-3, mask, 1e-4, sgs, case["weno"])
        else:
            u, v = _predict(u, v, 0.3 * H, 1e-3, mask.double(),
                            torch.sigmoid(-sdf.double() / (0.1 * H)), 1e-4, sgs, weno=case["weno"])
        return {"u": u, "v": v, "sgs": sgs}
    if k == "pure":
        mask, sdf = (t.double() for t in _obstacle("cylinder", nx, ny))
        u, v = (t.double() for t in _flow(nx, ny, seed))
        u, v, p = _pure(u, v, 0.4 * H, 1.5e-3, mask, sdf, 1e-4, lambda b: _vcycles(b, case["cycles"]))
        return {"u": u, "v": v, "p": p}
    cfg = _config(case)
    mac = cfg.grid_type == "mac"
    mask, sdf = _obstacle("naca" if mac else "cylinders", nx, ny)
    u, v = (t.double() for t in _flow(nx, ny, seed, mac))
    for _ in range(_steps_of(case)):
        if not mac:
            u, v, p = _gui_cylinders(u, v, cfg.nu, mask.double(), sdf.double())
        elif k == "gui":
            u, v, p = _gui_mac(u, v, cfg.nu, mask,
                               lambda b: _vcycles(b, case["cycles"], mask.double()))
        else:
            u, v, p = _gui_mac(u, v, cfg.nu, mask, lambda b: _solve(_pin(b * mask.double())))
    return {"u": u, "v": v, "p": p}
