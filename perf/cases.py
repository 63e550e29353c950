"""Performance cases of pybella_gb300: the calls that a user of the framework makes,
over the range of sizes, dimensions, precisions and options they are made with.

Kinds (the sizes are those of the repository's workloads, tests and benchmark, or
odd ones between them):

* ``matvec``      one product with the 9-point operator (``LinearOperator.matvec``)
* ``plain``       iterations of the reference's BiCGStab without preconditioner
                  (``linalg.bicgstab``), FP64 or double-float; a few, since the recurrences
                  multiply any difference of rounding by about two per iteration
* ``background``  a solve with the background solve as preconditioner, re-derived
                  from the step's coefficients first (2D BiCGStab, 3D FGMRES)
* ``ensemble``    iterations of an uneven ensemble's solves in one launch
* ``forward``     the learned preconditioner's network
* ``gradients``   its parameter gradients
* ``transport``   the advection of one time step (both halves, all sweeps)
* ``projection``  the 2D drop-in for the reference's implicit projection, on its own host arrays
* ``step``        a whole 3D time step: both projections, the explicit parts, the advection.
                  ``p2_nodes`` is not compared: the 27-point operator leaves it undetermined by
                  the null space's hourglass families, which hold the FP32 preconditioner's
                  rounding; ``f`` holds the corrections by its gradient, which is determined

A flow's arrays are restored from a device copy at the start of a pass, as a time
step resets ``Sol`` to ``Sol0``, so that every pass advances the same state.
"""
import ctypes
import math
from types import SimpleNamespace as NS

import numpy as np
import torch

from pybella_gb300 import _lib, ensemble, learned, linalg, workloads
from pybella_gb300.second_projection import euler_backward_non_advective_impl_part
from pybella_gb300.spectral import BackgroundSolve
from pybella_gb300.time_update import DeviceStep3D

FIELDS = ("rho", "rhou", "rhov", "rhow", "rhoY", "rhoX")
GAMM, MSQ, GRAV = 1.4, 100.0 / (287.4 * 300.0), 10.0 * 10000.0 / (287.4 * 300.0)
F64 = dict(dtype=torch.float64, device="cuda")


def listed():
    return [
        # the operator of the rising bubble's own grid, once: latency
        {"name": "matvec 161x81", "kind": "matvec", "cx": 160, "cy": 80},
        # the reference's solver on the reference's own grid
        {"name": "plain 2D fp64 161x81", "kind": "plain", "nx": 161, "ny": 81, "precision": "fp64", "maxiter": 16},
        # the stratified standalone solve, double-float
        {"name": "plain 2D df64 2049x1025", "kind": "plain", "nx": 2049, "ny": 1025, "precision": "df64",
         "maxiter": 16},
        # the same stratified systems as a time step solves them
        {"name": "background 2D 2049x1025", "kind": "background", "nd": 2, "nx": 2049, "ny": 1025, "nz": 1},
        {"name": "background 3D 257x129x257", "kind": "background", "nd": 3, "nx": 257, "ny": 129, "nz": 257},
        # the 48 rising-bubble members of three grids
        {"name": "ensemble 48", "kind": "ensemble", "cx": 160, "cy": 80, "per_grid": 16, "maxiter": 8},
        # the network on the 3D system, and a training window's gradients
        {"name": "forward 257x129x257", "kind": "forward", "nx": 257, "ny": 129, "nz": 257},
        {"name": "gradients 48x48x48", "kind": "gradients", "nx": 48, "ny": 48, "nz": 48},
        # transport: the rising bubble's grid, and the 3D system's
        {"name": "transport 2D 161x81", "kind": "transport", "nd": 2, "inx": 161, "iny": 81, "inz": 1, "odd": 1,
         "walls": False},
        {"name": "transport 3D 257x129x257", "kind": "transport", "nd": 3, "inx": 257, "iny": 129, "inz": 257,
         "odd": 0, "walls": False},
        # the reference's call on the reference's case, NumPy in and out
        {"name": "projection 2D 161x81", "kind": "projection", "nd": 2, "inx": 161, "iny": 81, "inz": 1},
        # the whole time step of the 3D system
        {"name": "step 3D 257x129x257", "kind": "step", "inx": 257, "iny": 129, "inz": 257, "odd": 1},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["matvec", "plain", "plain", "background", "ensemble", "forward", "gradients", "transport",
                       "transport", "projection", "step"])
    if kind == "matvec":
        cx = _log(rng, 40, 2048)
        return {"kind": kind, "cx": cx, "cy": max(17, cx // 2 + rng.randrange(-3, 4))}
    if kind == "plain":
        nx = _log(rng, 65, 1500)
        return {"kind": kind, "nx": nx, "ny": max(33, nx // 2 + rng.randrange(-5, 6)),
                "precision": rng.choice(["fp64", "df64"]), "maxiter": rng.randrange(6, 17)}
    if kind == "background" and rng.random() < 0.5:
        nx = 1 + (rng.choice([64, 128, 256, 512, 1024]) if rng.random() < 0.7 else 2 * _log(rng, 40, 300))
        return {"kind": kind, "nd": 2, "nx": nx, "ny": max(33, nx // 2 + rng.randrange(-8, 9)), "nz": 1}
    if kind == "background":
        n = [1 + rng.choice([32, 64, 128]) for _ in range(2)]
        return {"kind": kind, "nd": 3, "nx": n[0], "ny": rng.randrange(33, 100), "nz": n[1]}
    if kind == "ensemble":
        cx = 2 * rng.randrange(40, 90)
        return {"kind": kind, "cx": cx, "cy": cx // 2, "per_grid": rng.randrange(2, 13), "maxiter": rng.randrange(4, 10)}
    if kind == "forward":
        return {"kind": kind, "nx": _log(rng, 40, 257), "ny": _log(rng, 40, 140), "nz": _log(rng, 40, 257)}
    if kind == "gradients":
        n = 2 * rng.randrange(12, 40)
        return {"kind": kind, "nx": n, "ny": n, "nz": n}
    if kind == "transport" and rng.random() < 0.5:
        inx = _log(rng, 65, 1300)
        return {"kind": kind, "nd": 2, "inx": inx, "iny": max(33, inx // 2 + rng.randrange(-6, 7)), "inz": 1,
                "odd": rng.randrange(2), "walls": rng.random() < 0.25}
    if kind == "projection":
        inx = 1 + (rng.choice([64, 128, 256, 512]) if rng.random() < 0.6 else 2 * _log(rng, 40, 250))
        return {"kind": kind, "nd": 2, "inx": inx, "iny": max(33, inx // 2 + rng.randrange(-6, 7)), "inz": 1}
    inx = 1 + 2 * _log(rng, 16, 100)
    c = {"kind": kind, "inx": inx, "iny": max(17, inx // 2 + rng.randrange(-5, 6)),
         "inz": max(17, inx + 2 * rng.randrange(-6, 7))}
    if kind == "transport":
        return dict(c, nd=3, odd=rng.randrange(2), walls=rng.random() < 0.25)
    return dict(c, inz=1 + 2 * ((c["inz"] - 1) // 2), odd=rng.randrange(2))


# ---- flows ------------------------------------------------------------------
def _column(y, dy):
    """Isentropic hydrostatic background at heights y: rhoY0 and Y0."""
    Gamma = (GAMM - 1.0) / GAMM
    h = Gamma * GRAV
    pi_p, pi_m, pi = np.exp(-(y + 0.5 * dy) * h), np.exp(-(y - 0.5 * dy) * h), np.exp(-y * h)
    return pi ** (1.0 / (GAMM - 1.0)), -Gamma * GRAV * dy / (pi_p - pi_m)


def _flow(n, seed):
    """A warm bubble in a wavy wind on x, z in [-1, 1], y in [0, 1]: cell arrays with two ghost
    layers (a list in the order of FIELDS), the background columns and the spacings."""
    rng = np.random.default_rng(int(seed))
    nd = len(n)
    d = [(1.0 if k == 1 else 2.0) / (n[k] - 1.0) for k in range(nd)]
    x = [(0.0 if k == 1 else -1.0) + (np.arange(n[k] + 3) - 1.5) * d[k] for k in range(nd)]
    yn = (np.arange(n[1] + 4) - 2) * d[1]
    rhoY0, Y0 = _column(x[1], d[1])
    _, Y0n = _column(yn, d[1])
    X = [torch.tensor(x[k], **F64).reshape([-1 if q == k else 1 for q in range(nd)]) for k in range(nd)]
    amp, y0, x0 = rng.uniform(1.5, 2.5), rng.uniform(0.2, 0.4), rng.uniform(-0.05, 0.05)
    r2 = (X[0] - x0) ** 2 + (X[1] - y0) ** 2 + (X[2] ** 2 if nd == 3 else 0.0)
    r = torch.sqrt(r2) / 0.2
    pert = torch.where(r < 1.0, (amp / 300.0) * torch.cos(0.5 * math.pi * r) ** 2, torch.zeros_like(r))
    col = torch.tensor(rhoY0, **F64).reshape([1, -1] + [1] * (nd - 2))
    rhoY = col.expand(r.shape).contiguous()
    rho = rhoY / (1.0 + pert)

    def wave(a):
        ph = rng.uniform(0.0, 2.0 * math.pi, 3)
        w = torch.sin(math.pi * X[0] + ph[0]) * torch.cos(2.0 * math.pi * X[1] + ph[1])
        return a * (w + (0.5 * torch.sin(2.0 * math.pi * X[2] + ph[2]) if nd == 3 else 0.0))
    u = 0.1 + wave(0.05)
    v = wave(0.05) * torch.sin(math.pi * X[1])
    w = wave(0.05) if nd == 3 else wave(0.02)
    f = [rho, rho * u, rho * v, rho * w, rhoY, rho * (1.0 / (1.0 + pert) - 1.0 + wave(1e-3))]
    f = [a.expand(r.shape).contiguous() for a in f]
    S0c = torch.tensor(1.0 / Y0, **F64).reshape(col.shape).expand(r.shape)
    return NS(f=f, d=d, rhoY0=torch.tensor(rhoY0, **F64), S0n=torch.tensor(1.0 / Y0n, **F64), S0c=S0c,
              strat=torch.ones(n[1] + 3, **F64), elem_y=x[1], Y0n=Y0n, dt=0.3 * min(d) / 0.2)


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _dims(c):
    return [c["inx"], c["iny"]] + ([c["inz"]] if c.get("nd", 3) == 3 else [])


def _transport_state(c, seed):
    n = _dims(c)
    three = len(n) == 3
    fl = _flow(n, seed)
    ic = [k + 3 for k in n]
    a = _lib.Adv3D() if three else _lib.Adv2D()
    a.inx, a.iny, a.x_wall, a.y_wall = n[0], n[1], int(c["walls"]), 1
    a.dx, a.dy, a.g, a.gamm, a.is_compressible = fl.d[0], fl.d[1], GRAV, GAMM, 0
    shapes = [(ic[1], ic[0] + 1), (ic[0], ic[1] + 1)]
    if three:
        a.inz, a.z_wall, a.dz = n[2], int(c["walls"]), fl.d[2]
        shapes = [(ic[1], ic[2], ic[0] + 1), (ic[2], ic[0], ic[1] + 1), (ic[0], ic[1], ic[2] + 1)]
    f = [t.clone() for t in fl.f]
    for k, t in zip(FIELDS, f):
        setattr(a, k, _p(t))
    faces = [[torch.zeros(s, **F64) for _ in FIELDS] for s in shapes]
    for s, names in enumerate(("fx", "fy", "fz")[:len(n)]):
        for q in range(6):
            getattr(a, names)[q] = _p(faces[s][q])
    pwchi = torch.zeros(ic, **F64)
    a.hydro_rhoY0, a.strat_inv, a.pwchi = _p(fl.rhoY0), _p(fl.strat), _p(pwchi)
    return NS(lib=_lib.load(), a=a, f=f, f0=[torch.empty_like(t) for t in f], start=fl.f, faces=faces, pwchi=pwchi,
              keep=fl, nd=len(n), dt=fl.dt, odd=c["odd"])


def _run_transport(s):
    lib, a, st = s.lib, ctypes.byref(s.a), _stream()
    bd, fluxes, rk, advect = ((lib.bella_boundary3d, lib.bella_advective_fluxes3d, lib.bella_advect_rk3d,
                               lib.bella_advect3d) if s.nd == 3 else
                              (lib.bella_boundary2d, lib.bella_advective_fluxes2d, lib.bella_advect_rk2d,
                               lib.bella_advect2d))
    torch._foreach_copy_(s.f, s.start)
    _lib.check(bd(a, st), "boundary")
    torch._foreach_copy_(s.f0, s.f)
    _lib.check(fluxes(a, st), "advective_fluxes")
    _lib.check(rk(a, 0.5 * s.dt, st), "advect_rk")
    _lib.check(fluxes(a, st), "advective_fluxes")
    torch._foreach_copy_(s.f, s.f0)
    _lib.check(advect(a, s.dt, s.odd, st), "advect")
    return {"f": s.f, "mass": [q[4] for q in s.faces], "pwchi": s.pwchi}


def _objects(n, fl):
    """The flow in the reference's objects (host arrays): Sol, mpv, elem, node, ud, th."""
    Sol = NS(**{k: t.cpu().numpy() for k, t in zip(FIELDS, fl.f)})
    S0c = fl.S0c.cpu().numpy()
    mpv = NS(p2_nodes=np.zeros([k + 4 for k in n]), rhs=np.zeros([k + 2 for k in n]),
             HydroState=NS(rhoY0=fl.rhoY0.cpu().numpy(), get_S0c=lambda elem: S0c), HydroState_n=NS(S0=1.0 / fl.Y0n))
    node = NS(**dict(zip(("iicx", "iicy", "iicz", "dx", "dy", "dz"), (n + [1])[:3] + (fl.d + [1.0])[:3])),
              isc=tuple(k + 2 for k in n))
    ud = NS(bdry_type=["wrap", "symmetric", "wrap"], gravity_strength=[0.0, GRAV, 0.0], Msq=MSQ, nonhydrostasy=1.0,
            compressibility=0.0, is_compressible=0, coriolis_strength=np.zeros(3), u_wind_speed=0.0, v_wind_speed=0.0,
            w_wind_speed=0.0, stratification=lambda y: 1.0, tol=1e-10, max_iterations=1000)
    return Sol, mpv, NS(ndim=len(n), y=fl.elem_y), node, ud, NS(gamm=GAMM)


def _projection_state(c, seed):
    fl = _flow(_dims(c), seed)
    o = _objects(_dims(c), fl)
    return NS(o=o, start=[getattr(o[0], k).copy() for k in FIELDS], dt=0.5 * fl.dt)


def _run_projection(s):
    Sol, mpv, elem, node, ud, th = s.o
    for k, a in zip(FIELDS, s.start):
        np.copyto(getattr(Sol, k), a)
    mpv.p2_nodes[...] = 0.0
    euler_backward_non_advective_impl_part(Sol, mpv, elem, node, ud, th, 0.0, s.dt, 1.0, preconditioner="background")
    return {"f": [getattr(Sol, k) for k in FIELDS], "p2": mpv.p2_nodes, "rhs": mpv.rhs}


def _step_state(c, seed):
    n = _dims(c)
    fl = _flow(n, seed)
    run = DeviceStep3D(*_objects(n, fl), preconditioner="background")
    return NS(step=run, f=[run.f[k] for k in FIELDS] + [run.p2], start=fl.f + [torch.zeros_like(run.p2)], dt=fl.dt,
              odd=c["odd"])


def _run_step(s):
    torch._foreach_copy_(s.f, s.start)
    s.step.step(s.odd, s.dt)
    s.step.stats.clear()
    return {"f": s.f[:6], "rhs": s.step.rhs}


# ---- operators, solves and the network ---------------------------------------------
def _operator(c, seed):
    if c["nd"] == 2:
        w = workloads.stratified_2d(seed, c["nx"], c["ny"])
        return workloads.operator_2d(w), w
    w = workloads.stratified_3d(seed, c["nx"], c["ny"], c["nz"])
    return learned.operator_3d(w), w


def _member(c, seed):
    rng = np.random.default_rng(int(seed))
    return workloads.rising_bubble_member((c["cx"], c["cy"]), rng.normal(2.0, 0.2), rng.normal(0.0, 0.02))


def _vector(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1 + int(seed))
    return torch.randn(n, generator=g, **F64)


def _net(c, seed):
    shape = (c["nx"], c["ny"], c["nz"])
    net = learned.CNN(shape, block=2, mode="linear", skip=0.9)
    net.init(int(seed) % 2 ** 32, last_gain=0.1)
    n = shape[0] * shape[1] * shape[2]
    return net, shape, _vector(n, seed).float(), _vector(n, seed + 7).float()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "matvec":
        w = _member(case, seed)
        A = workloads.operator_2d(w)
        return NS(kind=kind, A=linalg.LinearOperator(A.shape, A), x=_vector(A.n, seed))
    if kind == "plain":
        A, w = _operator(dict(case, nd=2), seed)
        return NS(kind=kind, A=linalg.LinearOperator(A.shape, A), b=w["b"], maxiter=case["maxiter"],
                  precision=case["precision"])
    if kind == "background":
        A, w = _operator(case, seed)
        return NS(kind=kind, A=A, b=w["b"], bg=BackgroundSolve(A), three=case["nd"] == 3)
    if kind == "ensemble":
        rng = np.random.default_rng(int(seed))
        ms = [workloads.rising_bubble_member((q * case["cx"], q * case["cy"]), rng.normal(2.0, 0.2),
                                             rng.normal(0.0, 0.02)) for q in (1, 2, 4)
              for _ in range(case["per_grid"])]
        return NS(kind=kind, ops=[workloads.operator_2d(m) for m in ms], b=[m["b"] for m in ms],
                  maxiter=case["maxiter"])
    if kind in ("forward", "gradients"):
        net, shape, x, g = _net(case, seed)
        return NS(kind=kind, net=net, shape=shape, x=x, g=g)
    s = {"transport": _transport_state, "projection": _projection_state, "step": _step_state}[kind](case, seed)
    s.kind = kind
    return s


def run(s):
    if s.kind == "matvec":
        return s.A.matvec(s.x)
    if s.kind == "plain":
        return linalg.bicgstab(s.A, s.b, tol=1e-10, maxiter=s.maxiter, precision=s.precision)[0]
    if s.kind == "background":
        s.bg.update(s.A)
        if s.three:
            return s.A.solve(s.b, tol=1e-8, preconditioner=s.bg, method="fgmres", restart=30)[0]
        return linalg.bicgstab(s.A, s.b, tol=1e-8, maxiter=1000, M=s.bg)[0]
    if s.kind == "ensemble":
        return ensemble.solve_ensemble(s.ops, s.b, tol=1e-10, maxiter=s.maxiter, config=0)[0]
    if s.kind == "forward":
        return s.net.forward(s.x, s.shape, scale=1.0)
    if s.kind == "gradients":
        return s.net.gradients(s.x, s.g, s.shape)
    return {"transport": _run_transport, "projection": _run_projection, "step": _run_step}[s.kind](s)


# ---- what a pass cannot do without ----------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "matvec":
        n = (case["cx"] + 1) * (case["cy"] + 1)
        return {"bytes": 8 * 5 * n, "flops": 20 * n}
    if kind == "plain":
        n = case["nx"] * case["ny"]
        return {"bytes": 8 * 5 * n, "flops": case["maxiter"] * 62 * n}
    if kind == "background":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 8 * 5 * n, "flops": 10 * 120 * n}
    if kind == "ensemble":
        n = sum(case["per_grid"] * (q * case["cx"] + 1) * (q * case["cy"] + 1) for q in (1, 2, 4))
        return {"bytes": 8 * 5 * n, "flops": case["maxiter"] * 62 * n}
    if kind in ("forward", "gradients"):
        n = case["nx"] * case["ny"] * case["nz"]
        v = math.prod(-(-case[k] // 2) for k in ("nx", "ny", "nz"))
        f = 2 * 27 * v * (2 * 8 * 32 + 4 * 32 * 32)
        return {"bytes": 8 * n if kind == "forward" else 16 * n, "flops": f if kind == "forward" else 3 * f}
    n = math.prod(k + 3 for k in _dims(case))
    if kind == "transport":
        # both halves: the state in and out, the mass fluxes out, pwchi out
        nd = case["nd"]
        return {"bytes": 8 * n * (6 + 6 + nd + 1), "flops": n * (2 * nd * 45 + 4 * nd * 60)}
    if kind == "projection":
        return {"bytes": 8 * n * (6 + 6 + 1 + 1), "flops": 20 * 60 * n}
    return {"bytes": 8 * n * (7 + 7 + 1), "flops": 2 * 6 * 250 * n + 1000 * n}


# ---- 64-bit values ----------------------------------------------------------------------
def _exact_matvec(case, seed):
    """The 9-point operator (periodic x with the duplicated seam, walls in y) by its cell gradients."""
    w = _member(case, seed)
    nx, ny = w["nx"], w["ny"]
    p = _vector(nx * ny, seed).reshape(ny, nx)
    q = torch.zeros(ny + 2, nx + 2, **F64)
    q[1:-1, 1:-1] = p
    q[1:-1, 0], q[1:-1, -1] = p[:, -2], p[:, 1]
    h = [(w[k].reshape(ny + 1, nx + 1) * c.reshape(ny + 1, nx + 1)).clone()
         for k, c in (("hplusx", w["cor"][0]), ("hplusy", w["cor"][1]))]
    for t in h:
        t[0] = t[-1] = 0.0
    tl, tr, bl, br = q[:-1, :-1], q[:-1, 1:], q[1:, :-1], q[1:, 1:]
    fx = 0.5 * h[0] * ((tr - tl) + (br - bl)) / w["dx"] ** 2
    fy = 0.5 * h[1] * ((bl - tl) + (br - tr)) / w["dy"] ** 2
    y = 0.5 * ((fx[:-1, 1:] + fx[1:, 1:] - fx[:-1, :-1] - fx[1:, :-1])
               + (fy[1:, :-1] + fy[1:, 1:] - fy[:-1, :-1] - fy[:-1, 1:]))
    return (y * w["diag_inv"].reshape(ny, nx)).reshape(-1)


def _exact_boundary(f, s, nd, walls, rhoY0, g=GRAV):
    """Two ghost layers along axis s, in place."""
    at = lambda a, k: a.select(s, k)
    n = f[0].shape[s]
    if s == 1:
        for src, img in ((2, 1), (3, 0), (n - 3, n - 2), (n - 4, n - 1)):
            R = [at(a, src).clone() for a in f]
            Yr = R[4] / R[0]
            rY = torch.full_like(R[0], float(rhoY0[img]))
            new = [rY, rY * R[1] / R[0], -R[2] * Yr, rY * R[3] / R[0], rY, rY * R[5] / R[0]]
            for a, t in zip(f, new):
                at(a, img).copy_(t)
        return
    for q, a in enumerate(f):
        if not walls:
            for img, src in ((0, n - 4), (1, n - 3), (n - 2, 2), (n - 1, 3)):
                at(a, img).copy_(at(a, src).clone())
        elif q != 3:
            for img, src in ((1, 2), (0, 3), (n - 2, n - 3), (n - 1, n - 4)):
                at(a, img).copy_((-1.0 if q == 2 else 1.0) * at(a, src).clone())


def _exact_mass(f, nd):
    """Face mass fluxes per axis, (..., faces of the axis at its place), zero on the outer ones."""
    out = []
    for s in range(nd):
        m = f[4] * f[1 + s] / f[0]
        w = m.narrow(s, 0, m.shape[s] - 1) + m.narrow(s, 1, m.shape[s] - 1)
        for t in range(nd):
            if t != s:
                k = w.shape[t] - 2
                w = 0.5 * w.narrow(t, 0, k) + w.narrow(t, 1, k) + 0.5 * w.narrow(t, 2, k)
        w = w / (4.0 if nd == 2 else 8.0)
        shape = [k + (1 if t == s else 0) for t, k in enumerate(f[0].shape)]
        F = torch.zeros(shape, **F64)
        F[tuple(slice(1, -1) for _ in range(nd))] = w
        out.append(F)
    return out


def _exact_flux(f, F, s, nd, lam):
    """Upwind fluxes through every face of axis s (the outer ones zero); f[4]'s flux is the mass flux."""
    N = f[0].shape[s]
    P = [f[1] / f[0], f[2] / f[0], f[3] / f[0], f[5] / f[0], f[0] / f[4]]           # u, v, w, X, 1/Y
    U = torch.zeros_like(f[0])
    inner = tuple(slice(1, -1) for _ in range(nd))
    U[inner] = (0.5 * (F.narrow(s, 0, N) + F.narrow(s, 1, N)) / f[4])[inner]
    m = F.narrow(s, 1, N - 1)
    left = (m > 0).double() + 0.5 * (m == 0).double()
    face = []
    for q in P:
        S = torch.zeros_like(q)
        S.narrow(s, 1, N - 2).copy_(0.5 * (q.narrow(s, 2, N - 2) - q.narrow(s, 0, N - 2)))
        face.append(((q + 0.5 * S * (1.0 - lam * U)).narrow(s, 0, N - 1),
                     (q - 0.5 * S * (1.0 + lam * U)).narrow(s, 1, N - 1)))
    out = []
    for k in (None, 0, 1, 2, "mass", 3):
        if k == "mass":
            out.append(F)
            continue
        L, R = (1.0, 1.0) if k is None else face[k]
        G = torch.zeros_like(F)
        G.narrow(s, 1, N - 1).copy_(m * (left * face[4][0] * L + (1.0 - left) * face[4][1] * R))
        out.append(G)
    return out


def _exact_update(f, fl, s, lam):
    N = f[0].shape[s]
    for a, G in zip(f, fl):
        a += lam * (G.narrow(s, 0, N) - G.narrow(s, 1, N))


def _exact_transport(case, seed):
    n = _dims(case)
    nd, fl = len(n), _flow(n, seed)
    bd = lambda s: _exact_boundary(f, s, nd, case["walls"], fl.rhoY0)
    f = fl.f
    for s in range(nd):
        bd(s)
    f0 = [a.clone() for a in f]
    F = _exact_mass(f, nd)
    h, flux = 0.5 * fl.dt, []
    for s in range(nd):
        bd(s)
        flux.append(_exact_flux(f, F[s], s, nd, 0.0))
        bd(s)
    for s in range(nd):
        _exact_update(f, flux[s], s, h / fl.d[s])
    N = f[0].shape[1]
    pwchi = h / fl.d[1] * (flux[1][5].narrow(1, 0, N) - flux[1][5].narrow(1, 1, N))
    del flux
    for s in range(nd):
        bd(s)
    F = _exact_mass(f, nd)
    f = f0
    order = list(range(nd)) + list(range(nd - 1, -1, -1))
    for s in (order if case["odd"] else order[nd:] + order[:nd]):
        bd(s)
        _exact_update(f, _exact_flux(f, F[s], s, nd, h / fl.d[s]), s, h / fl.d[s])
        bd(s)
    for s in range(nd):
        bd(s)
    line = [(1, 0), (0, 1)] if nd == 2 else [(1, 2, 0), (2, 0, 1), (0, 1, 2)]
    return {"f": f, "mass": [F[s].permute(line[s]) for s in range(nd)], "pwchi": pwchi}


def _exact_forward(case, seed):
    """0.9 x + the six linear 3x3x3 convolutions on the grid of 2x2x2 node blocks, in 64 bits."""
    shape = (case["nx"], case["ny"], case["nz"])
    net, _, x, _ = _net(case, seed)
    p = torch.tensor(net.get_params(), **F64)
    c = [-(-k // 2) for k in shape]
    a = torch.zeros([2 * k for k in c], **F64)
    a[:shape[0], :shape[1], :shape[2]] = x.double().reshape(shape)
    a = a.reshape(c[0], 2, c[1], 2, c[2], 2).permute(0, 2, 4, 1, 3, 5).reshape(*c, 8)
    at = 0
    for cin, cout in ((8, 32), (32, 32), (32, 32), (32, 32), (32, 32), (32, 8)):
        W = p[at:at + 27 * cin * cout].reshape(27, cin, cout)
        at += 27 * cin * cout + cout
        q = torch.zeros([k + 2 for k in c] + [cin], **F64)
        q[1:-1, 1:-1, 1:-1] = a
        a = torch.zeros(*c, cout, **F64)
        for t in range(27):
            i, j, k = t // 9, t // 3 % 3, t % 3
            a += q[i:i + c[0], j:j + c[1], k:k + c[2]] @ W[t]
    a = a.reshape(*c, 2, 2, 2).permute(0, 3, 1, 4, 2, 5).reshape([2 * k for k in c])
    return a[:shape[0], :shape[1], :shape[2]].reshape(-1) + 0.9 * x.double()


def exact(case, seed):
    """None for the solves: what they return is an iterate, or a solution to a tolerance."""
    fn = {"matvec": _exact_matvec, "transport": _exact_transport, "forward": _exact_forward}.get(case["kind"])
    return fn(case, seed) if fn else None
