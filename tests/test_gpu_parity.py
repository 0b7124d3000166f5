"""GPU parity: every golden fixture (the reference's own source run in float64)
reproduced by the CUDA path through the C ABI, in FP32.

Tolerance: max|gpu - ref| / max|ref| <= 1e-5 for velocity and pressure
(the FP32 bar).  The one exception is the dynamic Smagorinsky model, whose
bound is the distance of the reference's own algorithm evaluated in FP32 from
its FP64 run (test_les)."""
import numpy as np
import pytest

from conftest import golden

pytestmark = pytest.mark.gpu
TOL = 1e-5


def rel(a, b):
    a = a.detach().double().cpu().numpy() if hasattr(a, "detach") else np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def T(x):
    import torch
    return torch.as_tensor(np.ascontiguousarray(x, dtype=np.float32), device="cuda")


@pytest.mark.parametrize("name", ["mg_64x32", "mg_128x48"])
def test_multigrid_parity(cuda_lib, name):
    import aerojax_gb300 as aj
    g = golden(name)
    p = aj.poisson_multigrid(T(g["rhs"]), T(g["mask"]), float(g["dx"]), float(g["dy"]),
                             v_cycles=int(g["v_cycles"]))
    pm = aj.poisson_multigrid_mac(T(g["rhs"]), T(g["mask"]), float(g["dx"]), float(g["dy"]),
                                  v_cycles=int(g["v_cycles"]))
    assert rel(p, g["p"]) < TOL
    assert rel(pm, g["p_mac"]) < TOL


@pytest.mark.parametrize("nx,ny,guess", [(64, 32, True), (48, 80, False), (272, 48, False),
                                         (96, 2048, False), (1008, 368, True)])
def test_multigrid_parity_bands(cuda_lib, nx, ny, guess):
    """Grids that put all, some or only the lower levels of the V-cycle on the
    cluster, with bands that end inside the last blocks."""
    import aerojax_gb300 as aj
    from oracle import ref_np as R
    rng = np.random.default_rng(nx + ny)
    dx, dy = 0.02, 0.025
    rhs = rng.standard_normal((nx, ny)).astype(np.float32)
    mask = (rng.random((nx, ny)) > 0.05).astype(np.float32)
    p0 = rng.standard_normal((nx, ny)).astype(np.float32) * 1e-3 if guess else None
    for mac in (False, True):
        fn = aj.poisson_multigrid_mac if mac else aj.poisson_multigrid
        p, st = fn(T(rhs), T(mask), dx, dy, v_cycles=3, p0=T(p0) if guess else None,
                   return_stats=True)
        ref = R.poisson_multigrid(rhs.astype(np.float64), mask.astype(np.float64), dx, dy,
                                  v_cycles=3, mac=mac, p0=None if p0 is None else p0.astype(np.float64))
        assert rel(p, ref) < TOL, (mac, rel(p, ref))
        assert st["cycles"] == 3 and st["err"] == 0


@pytest.mark.parametrize("nx,ny", [(512, 256), (528, 272)])
def test_mac_step_wide(cuda_lib, nx, ny):
    """The right-hand side and the correction four columns a thread (from 2^17
    cells; whole and partial blocks of 128 columns), through a MAC step against
    the oracle; the fields one float off the 16-byte boundary take the kernels of
    a cell a thread and give the same bits."""
    import torch
    from aerojax_gb300.params import StepConfig
    from aerojax_gb300.solver import Plan, run_step
    from oracle import ref_np as R
    rng = np.random.default_rng(nx)
    f = lambda n, m, a, s: (a + s * rng.standard_normal((n, m))).astype(np.float32)
    u, v = f(nx + 1, ny, 1.0, 0.2), f(nx, ny + 1, 0.0, 0.2)
    mask = (rng.random((nx, ny)) > 0.02).astype(np.float32)
    cfg = StepConfig(nx=nx, ny=ny, dx=0.02, dy=0.025, nu=1e-3, grid_type="mac", variant="gui",
                     v_cycles=2, brinkman_eta=1e-3, dt=2e-3)
    outs = []
    for off in (0, 1):
        def place(a):
            t = torch.zeros(a.size + 4, device="cuda")[off:off + a.size].view(a.shape)
            t.copy_(torch.as_tensor(a))
            return t
        m = place(mask)
        plan = Plan(cfg, m.device)
        plan.prepare(m)
        out = tuple(place(np.zeros(s, np.float32)) for s in ((nx + 1, ny), (nx, ny + 1), (nx, ny)))
        outs.append([t.clone() for t in run_step(plan, place(u), place(v), m, out=out)])
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    d = lambda a: a.astype(np.float64)
    us, vs = R.rk_step_unified_mac(d(u), d(v), 2e-3, 1e-3, 0.02, 0.025, d(mask), U_inf=1.0,
                                   slip_walls=True, brinkman_eta=1e-3)
    p = d(outs[0][2].cpu().numpy())
    dpx = np.zeros((nx + 1, ny))
    dpx[1:-1] = (p[1:] - p[:-1]) / 0.02
    dpy = np.zeros((nx, ny + 1))
    dpy[:, 1:-1] = (p[:, 1:] - p[:, :-1]) / 0.025
    assert rel(outs[0][0][2:-2, 2:-2], (us - 2e-3 * dpx)[2:-2, 2:-2]) < TOL
    assert rel(outs[0][1][2:-2, 2:-2], (vs - 2e-3 * dpy)[2:-2, 2:-2]) < TOL


@pytest.mark.parametrize("nx,ny", [(7, 6), (31, 246), (160, 247), (309, 40), (611, 493)])
def test_dynamic_smagorinsky_strips(cuda_lib, nx, ny):
    """The dynamic model's strips of columns (one full, one column more, three)
    and runs of rows (2 to 6 a block, a partial last one), against the FP64
    oracle; on these fields the oracle in FP32 is within 1e-8 of C_d and
    5e-7 of the viscosity."""
    import aerojax_gb300 as aj
    from oracle import ref_np as R
    rng = np.random.default_rng(nx + ny)
    u, v = (rng.standard_normal((nx, ny)).astype(np.float32) for _ in range(2))
    got, cd = aj.dynamic_smagorinsky(T(u), T(v), 0.02, 0.03, 0.025)
    d = lambda a: a.astype(np.float64)
    want, cdr = R.dynamic_smagorinsky(d(u), d(v), 0.02, 0.03, 0.025)
    assert float(np.max(np.abs(cd.cpu().numpy() - cdr))) < 1e-6
    assert rel(got, want) < TOL


@pytest.mark.parametrize("hyper,fast,slip,flow", [(0.0, False, True, "von_karman"),
                                                  (0.05, False, False, "von_karman"),
                                                  (0.05, True, True, "von_karman"),
                                                  (0.02, False, True, "lid_driven_cavity")])
def test_predictor_collocated_wide(cuda_lib, hyper, fast, slip, flow):
    """The stage kernel that takes four columns a thread (grids of 2^17 cells
    and rows of a multiple of 4), its edge cells and partial blocks."""
    import aerojax_gb300 as aj
    from oracle import ref_np as R
    nx, ny = 517, 260
    rng = np.random.default_rng(5)
    f = lambda a, s: (a + s * rng.standard_normal((nx, ny))).astype(np.float32)
    u, v, sgs = f(1.0, 0.3), f(0.0, 0.3), np.abs(f(0.0, 1e-3))
    mask = (rng.random((nx, ny)) > 0.02).astype(np.float32)
    kw = dict(U_inf=1.1, nu_hyper_ratio=hyper, slip_walls=slip, fast_mode=fast,
              brinkman_eta=1e-3, flow_type=flow)
    us, vs = aj.rk_step_unified(T(u), T(v), 2e-3, 1e-2, 0.02, 0.025, T(mask), nu_sgs=T(sgs), **kw)
    d = lambda a: a.astype(np.float64)
    ur, vr = R.rk_step_unified(d(u), d(v), 2e-3, 1e-2, 0.02, 0.025, d(mask), nu_sgs=d(sgs), **kw)
    assert rel(us, ur) < TOL and rel(vs, vr) < TOL


def test_multigrid_parity_unaligned(cuda_lib):
    """A mask and a result that start on 4-byte boundaries only: the tiled
    kernels' pairs fall back to single cells and give the same bits."""
    import ctypes
    import torch
    import aerojax_gb300 as aj
    from aerojax_gb300._lib import check, lib
    nx, ny = 448, 304
    rng = np.random.default_rng(3)
    rhs = T(rng.standard_normal((nx, ny)))
    mask = T(rng.random((nx, ny)) > 0.05)
    cfg = aj.StepConfig(nx=nx, ny=ny, dx=0.02, dy=0.025, nu=1.0, grid_type="mac", variant="gui",
                        v_cycles=2)
    plan = aj.Plan(cfg, rhs.device)
    out = []
    for off in (0, 1):
        k = torch.zeros(nx * ny + 1, device="cuda")[off:off + nx * ny].copy_(mask.reshape(-1))
        p = torch.zeros(nx * ny + 1, device="cuda")[off:off + nx * ny]
        plan.prepare(k)
        check("aj_poisson_mg", lib().aj_poisson_mg(
            ctypes.byref(plan.params), rhs.data_ptr(), k.data_ptr(), None, p.data_ptr(),
            plan.ws.data_ptr(), plan.nbytes, None, torch.cuda.current_stream().cuda_stream))
        out.append(p.clone())
    assert torch.equal(*out) and float(out[0].abs().max()) > 0


@pytest.mark.parametrize("mac", [False, True])
def test_predictor_takes_each_calls_dt(cuda_lib, mac):
    """Calls that differ in their time step alone (they share a workspace), there
    and back, each against the oracle at its own dt."""
    import aerojax_gb300 as aj
    from oracle import ref_np as R
    nx, ny = 66, 38
    rng = np.random.default_rng(21)
    f = lambda n, m, a: (a + 0.1 * rng.standard_normal((n, m))).astype(np.float32)
    u, v = (f(nx + 1, ny, 1.0), f(nx, ny + 1, 0.0)) if mac else (f(nx, ny, 1.0), f(nx, ny, 0.0))
    mask = np.ones((nx, ny), np.float32)
    gpu = aj.rk_step_unified_mac if mac else aj.rk_step_unified
    ref = R.rk_step_unified_mac if mac else R.rk_step_unified
    d = lambda a: a.astype(np.float64)
    for dt in (1e-3, 4e-3, 1e-3):
        got = gpu(T(u), T(v), dt, 4e-3, 1 / 64, 1 / 48, T(mask), brinkman_eta=1e-3)
        want = ref(d(u), d(v), dt, 4e-3, 1 / 64, 1 / 48, d(mask), brinkman_eta=1e-3)
        assert rel(got[0], want[0]) < TOL
        assert rel(got[1], want[1]) < TOL


def test_plan_takes_each_configurations_dt(cuda_lib):
    """A step through get_plan's plan runs with the dt of the configuration asked
    for, whichever came before it."""
    import aerojax_gb300 as aj
    u, v, mask = T(np.ones((64, 48))), T(np.zeros((64, 48))), T(np.ones((64, 48)))
    for dt in (2e-3, 3e-3, 2e-3):
        plan = aj.get_plan(aj.StepConfig(nx=64, ny=48, dx=0.02, dy=0.02, nu=1e-3, dt=dt), u.device)
        plan.prepare(mask)
        aj.run_step(plan, u, v, mask)
        assert plan.stats()["dt"] == np.float32(dt)


@pytest.mark.parametrize("nx,ny,step,count", [(288, 48, 16, 17), (448, 304, 4, 6)])
@pytest.mark.parametrize("mac", [False, True])
def test_rhs_norm_is_a_double_sum(cuda_lib, nx, ny, step, count, mac):
    """The V-cycle's norms (the whole solve on the cluster; one block of the tiled
    level-0 kernel) are FP64 sums of the warps' totals: 1, 2^-24 and a few times
    2^-52 from as many warps add up without a rounding, which a pair of FP32
    numbers cannot hold."""
    import aerojax_gb300 as aj
    rhs = np.zeros((nx, ny), np.float32)
    rhs[step * np.arange(count), 5] = [1.0, 2.0 ** -12] + [2.0 ** -26] * (count - 2)
    fn = aj.poisson_multigrid_mac if mac else aj.poisson_multigrid
    _, st = fn(T(rhs), T(np.ones((nx, ny))), 0.02, 0.025, v_cycles=1, return_stats=True)
    assert st["rhs_norm"] == np.sqrt(1.0 + 2.0 ** -24 + (count - 2) * 2.0 ** -52)


@pytest.mark.parametrize("nx,ny", [(2048, 512), (64, 8192), (64, 32768)])
def test_multigrid_parity_wide_coarsest(cuda_lib, nx, ny):
    """Two levels below the finest on grids whose coarsest bands do not fit the
    V-cycle's cluster: the coarsest sweeps on a cluster of their own, and, where
    not even that holds them (64x32768), a launch a sweep."""
    import aerojax_gb300 as aj
    from oracle import ref_np as R
    rng = np.random.default_rng(nx + ny)
    dx, dy = 0.02, 0.025
    rhs = rng.standard_normal((nx, ny)).astype(np.float32)
    mask = (rng.random((nx, ny)) > 0.05).astype(np.float32)
    d = lambda a: a.astype(np.float64)
    for mac in (False, True):
        fn = aj.poisson_multigrid_mac if mac else aj.poisson_multigrid
        p, st = fn(T(rhs), T(mask), dx, dy, levels=2, v_cycles=2, return_stats=True)
        ref = R.poisson_multigrid(d(rhs), d(mask), dx, dy, levels=2, v_cycles=2, mac=mac)
        assert rel(p, ref) < TOL, (mac, rel(p, ref))
        assert st["cycles"] == 2 and st["err"] == 0


@pytest.mark.parametrize("name", ["rk3", "rk2", "rk3_hyper", "rk3_field"])
def test_predictor_collocated(cuda_lib, name):
    import aerojax_gb300 as aj
    g = golden("pred_" + name)
    field = g["nu_sgs"].shape != (1, 1)
    us, vs = aj.rk_step_unified(T(g["u"]), T(g["v"]), float(g["dt"]), 0.01 if field else float(g["nu"]),
                                float(g["dx"]), float(g["dy"]), T(g["mask"]), sdf=T(g["sdf"]),
                                U_inf=float(g["U"]), nu_sgs=T(g["nu_sgs"]) if field else None,
                                nu_hyper_ratio=float(g["hyper"]), fast_mode=bool(g["fast"]),
                                brinkman_eta=float(g["eta"]), double_count=field)
    assert rel(us, g["u_star"]) < TOL
    assert rel(vs, g["v_star"]) < TOL


@pytest.mark.parametrize("name", ["mac_rk3", "mac_rk2_les_hyper"])
def test_predictor_mac(cuda_lib, name):
    import aerojax_gb300 as aj
    g = golden("pred_" + name)
    field = g["nu_sgs"].shape != (1, 1)
    us, vs = aj.rk_step_unified_mac(T(g["u"]), T(g["v"]), float(g["dt"]), float(g["nu"]),
                                    float(g["dx"]), float(g["dy"]), T(g["mask"]), U_inf=float(g["U"]),
                                    nu_sgs=T(g["nu_sgs"]) if field else None,
                                    nu_hyper_ratio=float(g["hyper"]), fast_mode=bool(g["fast"]),
                                    brinkman_eta=float(g["eta"]))
    assert rel(us, g["u_star"]) < TOL
    assert rel(vs, g["v_star"]) < TOL


@pytest.mark.parametrize("shape,slip,les", [((100, 68), True, True), ((70, 44), False, True),
                                             ((34, 8), True, False), ((256, 64), True, True)])
def test_predictor_mac_tile(cuda_lib, shape, slip, les):
    """The MAC RK3 predictor on grids the one-kernel tile path covers (nx
    even, ny a multiple of 4), whole and partial 32x32 tiles, slip and
    no-slip walls, with and without eddy viscosity, against the oracle."""
    import aerojax_gb300 as aj
    from oracle import ref_np as R
    nx, ny = shape
    rng = np.random.default_rng(nx * ny)
    dx, dy, dt, nu, eta = 1 / 64, 1 / 48, 2e-3, 4e-3, 1e-3
    u = (1 + 0.1 * rng.standard_normal((nx + 1, ny))).astype(np.float32).astype(np.float64)
    v = (0.1 * rng.standard_normal((nx, ny + 1))).astype(np.float32).astype(np.float64)
    X, Y = np.meshgrid((np.arange(nx) + .5) * dx, (np.arange(ny) + .5) * dy, indexing="ij")
    mask = R.mask_from_sdf(R.sdf_cylinder(X, Y, 0.4 * nx * dx, 0.5 * ny * dy, 3 * dx), 0.5 * dx)
    mask = mask.astype(np.float32).astype(np.float64)
    nsg = (1e-3 * rng.random((nx, ny))).astype(np.float32).astype(np.float64) if les else None
    ur, vr = R.rk_step_unified_mac(u, v, dt, nu, dx, dy, mask, nu_sgs=nsg, slip_walls=slip,
                                   brinkman_eta=eta)
    ug, vg = aj.rk_step_unified_mac(T(u), T(v), dt, nu, dx, dy, T(mask),
                                    nu_sgs=T(nsg) if les else None, slip_walls=slip,
                                    brinkman_eta=eta)
    assert rel(ug, ur) < TOL
    assert rel(vg, vr) < TOL


def test_les(cuda_lib):
    import aerojax_gb300 as aj
    g = golden("les")
    c = aj.constant_smagorinsky(T(g["u"]), T(g["v"]), float(g["dx"]), float(g["dy"]),
                                float(g["delta"]), 0.17)
    d, cd = aj.dynamic_smagorinsky(T(g["u"]), T(g["v"]), float(g["dx"]), float(g["dy"]),
                                   float(g["delta"]))
    assert rel(c, g["nu_const"]) < TOL
    # C_d = <LM>/(<MM>+1e-8): L_ij = filter(u_i)filter(u_j) - filter(u_i u_j)
    # cancels to ~1e-4 of its terms, so the reference's own algorithm
    # evaluated in FP32 departs from its FP64 run by ~1.2e-4 on this field.
    # The GPU must be no further from FP64 than that FP32 evaluation.
    d32, cd32 = _dynamic_fp32(g)
    assert rel(cd, g["cd"]) <= max(TOL, 2.0 * rel(cd32, g["cd"]))
    assert rel(d, g["nu_dyn"]) <= max(TOL, 2.0 * rel(d32, g["nu_dyn"]))
    assert rel(d32, g["nu_dyn"]) > 10 * TOL     # the bound is the FP32 evaluation's, not 1e-5


def _dynamic_fp32(g):
    """The oracle's dynamic Smagorinsky in FP32 arithmetic (the reference's
    default precision, solver/config.py:28) on the fixture's inputs."""
    from oracle import ref_np as R
    f = np.float32
    return R.dynamic_smagorinsky(g["u"].astype(f), g["v"].astype(f), f(g["dx"]), f(g["dy"]),
                                 f(g["delta"]))


def test_step_pure(cuda_lib):
    import aerojax_gb300 as aj
    g = golden("step_pure")
    st = aj.SimState(u=T(g["u"]), v=T(g["v"]), p=None, u_prev=None, v_prev=None, c=None,
                     dt=float(g["dt"]), iteration=0)
    out = aj.step_pure(st, T(g["mask"]), T(g["sdf"]), float(g["dx"]), float(g["dy"]), float(g["nu"]),
                       float(g["U"]), v_cycles=int(g["v_cycles"]), brinkman_eta=float(g["eta"]))
    assert out.iteration == 1
    assert rel(out.u, g["u_new"]) < TOL
    assert rel(out.v, g["v_new"]) < TOL
    assert rel(out.p, g["p"]) < TOL


@pytest.mark.parametrize("name", ["gui_col_les", "gui_col_dyn", "gui_col_plain", "gui_mac_les",
                                  "gui_mac_plain"])
def test_step_gui(cuda_lib, name):
    import aerojax_gb300 as aj
    g = golden("step_" + name)
    mac = "mac" in name
    nx, ny = g["mask"].shape
    h = aj.StepHandler(nx, ny, float(g["dx"]), float(g["dy"]), float(g["nu"]), float(g["U"]),
                       grid_type="mac" if mac else "collocated", use_les=bool(g["use_les"]),
                       les_model="dynamic_smagorinsky" if int(g["dynamic"]) else "smagorinsky",
                       smagorinsky_constant=float(g["cs"]), nu_hyper_ratio=float(g["hyper"]),
                       brinkman_eta=float(g["eta"]), multigrid_v_cycles=int(g["v_cycles"]),
                       sdf=None if mac else T(g["sdf"]), dt=float(g["dt"]))
    u, v, p = h._step(T(g["u"]), T(g["v"]), T(g["mask"]))
    if int(g["dynamic"]):
        # dynamic C_d (see test_les): bounded by the reference's own step
        # evaluated in FP32 from the same inputs
        from oracle import ref_np as R
        f = np.float32
        r32 = R.step_gui(g["u"].astype(f), g["v"].astype(f), g["mask"].astype(f), f(g["dt"]),
                         sdf=None if mac else g["sdf"].astype(f), dx=f(g["dx"]), dy=f(g["dy"]),
                         nu=f(g["nu"]), U_inf=f(g["U"]), grid_type="mac" if mac else "collocated",
                         use_les=True, les_model="dynamic_smagorinsky",
                         smagorinsky_constant=f(g["cs"]), nu_hyper_ratio=f(g["hyper"]),
                         brinkman_eta=f(g["eta"]), v_cycles=int(g["v_cycles"]))
        for got, key, ref32 in ((u, "u_new", r32[0]), (v, "v_new", r32[1]), (p, "p", r32[2])):
            assert rel(got, g[key]) <= max(TOL, 2.0 * rel(ref32, g[key])), key
        return
    assert rel(u, g["u_new"]) < TOL
    assert rel(v, g["v_new"]) < TOL
    assert rel(p, g["p"]) < TOL


def test_cfl(cuda_lib):
    import aerojax_gb300 as aj
    g = golden("cfl")
    a = aj.compute_cfl_timestep(T(g["u"]), T(g["v"]), float(g["dx"]), float(g["dy"]), float(g["nu"]),
                                cfl_target=0.5, dt_min=1e-5, dt_max=0.05)
    b = aj.compute_cfl_timestep(T(g["um"]), T(g["vm"]), float(g["dx"]), float(g["dy"]),
                                float(g["nu"]), cfl_target=0.5, dt_min=1e-5, dt_max=0.05)
    assert float(a.item()) == pytest.approx(float(g["dt"]), rel=1e-6)
    assert float(b.item()) == pytest.approx(float(g["dt_mac"]), rel=1e-6)


def test_geometry(cuda_lib):
    import aerojax_gb300 as aj
    from oracle import ref_np as R
    g = golden("geometry")
    nx, ny = g["X"].shape
    lx, ly = float(g["X"][-1, 0]), float(g["Y"][0, -1])
    eps = 0.05 * lx / nx
    for kind, geo, key in [("naca4", (1.5, 10.0, 1.5, 1.5, 0.0, 0.0, 0.12), "sdf_naca0012"),
                           ("naca4", (1.5, 5.0, 1.5, 1.5, 0.02, 0.4, 0.12), "sdf_naca2412"),
                           ("cyl3_row", (2.0, 1.5, 0.5, 0.8), "sdf_three")]:
        mask, sdf = aj.make_geometry(kind, nx, ny, lx, ly, geo, eps)
        ref = g[key]
        assert np.nanmax(np.abs(sdf.cpu().numpy() - ref)) < 1e-6
        mref = R.mask_from_sdf(ref, eps)
        assert np.max(np.abs(mask.cpu().numpy() - mref)) < 1e-5
    # the triangle of three cylinders has no reference counterpart: the oracle's
    # SDF (sdf_three_cylinders_triangle) on the fixture's grid
    X, Y = g["X"], g["Y"]
    geo = (2.0, 1.5, 0.5, 0.8)
    mask, sdf = aj.make_geometry("cyl3_tri", nx, ny, lx, ly, geo, eps)
    ref = R.sdf_three_cylinders_triangle(X, Y, *geo)
    assert np.max(np.abs(sdf.cpu().numpy() - ref)) < 1e-6
    assert np.max(np.abs(mask.cpu().numpy() - R.mask_from_sdf(ref, eps))) < 1e-5


def test_shape_error_like_reference(cuda_lib):
    import aerojax_gb300 as aj
    import torch
    rhs = torch.zeros((100, 64), device="cuda")
    with pytest.raises(ValueError):
        aj.poisson_multigrid(rhs, torch.ones_like(rhs), 0.01, 0.01)


def test_step_gui_no_slip_walls_against_oracle(cuda_lib):
    """The collocated GUI step with no-slip walls (slip_walls=False) and
    hyperviscosity, which the golden fixtures (slip walls) do not cover,
    against the oracle's step_gui on a 96x80 cylinder case."""
    import aerojax_gb300 as aj
    from oracle import ref_np as R
    nx, ny, dx, dt = 96, 80, 0.05, 0.004
    rng = np.random.default_rng(21)
    X, Y = np.meshgrid((np.arange(nx) + 0.5) * dx, (np.arange(ny) + 0.5) * dx, indexing="ij")
    sdf = R.sdf_cylinder(X, Y, 1.4, 2.0, 0.4)
    mask = R.mask_from_sdf(sdf, 0.5 * dx)
    u = 1.0 + 0.1 * rng.standard_normal((nx, ny))
    v = 0.1 * rng.standard_normal((nx, ny))
    kw = dict(nu_hyper_ratio=0.05, slip_walls=False, brinkman_eta=1e-3)
    ur, vr, pr = R.step_gui(u, v, mask, dt, sdf=sdf, dx=dx, dy=dx, nu=0.02, U_inf=1.0,
                            v_cycles=3, **kw)
    h = aj.StepHandler(nx, ny, dx, dx, 0.02, 1.0, grid_type="collocated", use_les=False,
                       multigrid_v_cycles=3, sdf=T(sdf), dt=dt, **kw)
    ug, vg, pg = h._step(T(u), T(v), T(mask))
    assert rel(ug, ur) < TOL
    assert rel(vg, vr) < TOL
    assert rel(pg, pr) < TOL


@pytest.mark.parametrize("tag", ["ldc", "tg"])
def test_other_flow_types(cuda_lib, tag):
    """Lid-driven cavity and Taylor-Green through the C ABI against the
    reference's own results (fixtures flow_*): the parity multigrid on both
    grids (mean subtraction and centre pin; the wrapped residual), step_pure,
    and the GUI step on the collocated and the MAC grid."""
    import aerojax_gb300 as aj
    g = golden(f"flow_mg_{tag}")
    flow = str(g["flow"])
    p = aj.poisson_multigrid(T(g["rhs"]), T(g["mask"]), float(g["dx"]), float(g["dy"]),
                             v_cycles=int(g["v_cycles"]), flow_type=flow)
    pm = aj.poisson_multigrid_mac(T(g["rhs"]), T(g["mask"]), float(g["dx"]), float(g["dy"]),
                                  v_cycles=int(g["v_cycles"]), flow_type=flow)
    assert rel(p, g["p"]) < TOL, rel(p, g["p"])
    assert rel(pm, g["p_mac"]) < TOL, rel(pm, g["p_mac"])
    g = golden(f"flow_step_pure_{tag}")
    st = aj.SimState(u=T(g["u"]), v=T(g["v"]), p=None, u_prev=None, v_prev=None, c=None,
                     dt=float(g["dt"]), iteration=0)
    out = aj.step_pure(st, T(g["mask"]), T(g["sdf"]), float(g["dx"]), float(g["dy"]),
                       float(g["nu"]), float(g["U"]), v_cycles=int(g["v_cycles"]),
                       brinkman_eta=float(g["eta"]), flow_type=flow)
    for got, key in ((out.u, "u_new"), (out.v, "v_new"), (out.p, "p")):
        assert rel(got, g[key]) < TOL, (key, rel(got, g[key]))
    for grid in ("col", "mac"):
        g = golden(f"flow_gui_{grid}_{tag}")
        mac = grid == "mac"
        nx, ny = g["mask"].shape
        h = aj.StepHandler(nx, ny, float(g["dx"]), float(g["dy"]), float(g["nu"]),
                           float(g["U"]), grid_type="mac" if mac else "collocated",
                           flow_type=flow, use_les=True, les_model="smagorinsky",
                           smagorinsky_constant=float(g["cs"]), nu_hyper_ratio=float(g["hyper"]),
                           brinkman_eta=float(g["eta"]), multigrid_v_cycles=int(g["v_cycles"]),
                           sdf=None if mac else T(g["sdf"]), dt=float(g["dt"]))
        u, v, p = h._step(T(g["u"]), T(g["v"]), T(g["mask"]))
        for got, key in ((u, "u_new"), (v, "v_new"), (p, "p")):
            assert rel(got, g[key]) < TOL, (grid, key, rel(got, g[key]))
