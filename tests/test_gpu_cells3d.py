"""The 3D projection's cell and node kernels at the edges of their tiles (8 x 32 in y and z,
segments along x), with and without Coriolis forces, walls, wind and compressibility: the
explicit parts against the host build of bella_expl3d.cuh (tests/expl3d_host.cpp), the
coefficients, the diagonal, the divergence and the correction of the implicit part against
the oracle's pieces, with the solve stopped before its first iteration.

Tolerance: each value is a sum of terms no larger than its field's maximum from fewer than
100 FP64 operations (100 eps = 2e-14 of it) in at most four passes: 1e-12 of the maximum; the
divergence is a difference of momenta over a spacing, whose rounding is eps times the momenta
over the spacing, and the operator's action one of the vector's entries."""
import ctypes

import numpy as np
import pytest

from test_expl3d_host import FIELDS, _geom, _ptr, host_lib  # noqa: F401

pytestmark = pytest.mark.gpu

SHAPES = [(5, 5, 5), (13, 9, 11), (7, 38, 70), (70, 6, 31), (35, 17, 64)]
REGIMES = {"plain": ((False, True, False), (0.0, 0.0, 0.0), (0.0, 0.0, 0.0), False),
           "wind": ((False, True, True), (0.0, 0.0, 0.0), (0.5, 0.1, 0.2), False),
           "cor": ((True, True, False), (3.0, 2.0, 1.0), (0.5, 0.0, 0.2), True)}


def _inputs(shape, regime, seed=5):
    from oracle import cases, proj3d as o3
    walls, cor, wind, comp = REGIMES[regime]
    bdry = tuple(o3.WALL if w else o3.PERIODIC for w in walls)
    grid, prm, Sol, p2, hn, hc, sf = cases.bubble_3d(*shape, seed=seed, bdry=bdry, coriolis=cor, compressible=comp)
    p2[...] = 0.05 * np.random.default_rng(6).standard_normal(p2.shape)
    hn = dict(hn, S0=hn["S0"] * (1.0 - 0.1 * np.linspace(0.0, 1.0, hn["S0"].size)))       # stratified
    Sol["rhoX"] = Sol["rho"] * 0.01 * np.random.default_rng(7).standard_normal(Sol["rho"].shape)
    return grid, prm, Sol, p2, hn, hc, sf, wind


def _args(cls, grid, prm, dt, keep):
    a = cls()
    a.inx, a.iny, a.inz = grid.inx, grid.iny, grid.inz
    a.x_wall, a.y_wall, a.z_wall = (int(grid.wall(d)) for d in range(3))
    a.dx, a.dy, a.dz, a.dt = grid.dx, grid.dy, grid.dz, dt
    a.Msq, a.g, a.gamm, a.nonhydro, a.compressibility = prm.Msq, prm.g, prm.gamm, prm.nonhydro, prm.compressibility
    a.is_compressible, a.div_sign_2d = prm.is_compressible, 0
    for q in range(3):
        a.coriolis[q] = float(prm.coriolis[q])
    for k, t in keep.items():
        if k in dict(cls._fields_):
            setattr(a, k, ctypes.c_void_p(t.data_ptr()))
    return a


def _dev(arrays):
    import torch
    return {k: torch.tensor(np.ascontiguousarray(v, dtype=np.float64), device="cuda") for k, v in arrays.items()}


def _close(got, ref, scale=None, what=""):
    got = got.cpu().numpy() if hasattr(got, "cpu") else got
    s = np.abs(ref).max() if scale is None else scale
    assert np.abs(got - ref).max() <= 1e-12 * max(s, 1e-300), (what, np.abs(got - ref).max(), s)


@pytest.mark.parametrize("regime", sorted(REGIMES))
@pytest.mark.parametrize("shape", SHAPES)
def test_explicit_parts_match_the_host_build(host_lib, shape, regime):  # noqa: F811
    import torch
    from pybella_gb300 import _lib
    grid, prm, Sol, p2, hn, hc, sf, wind = _inputs(shape, regime)
    S0c = np.broadcast_to(hc["S0"][None, :, None], grid.elem_sc).copy()
    dt = 0.02
    base = dict({k: Sol[k] for k in FIELDS}, p2=p2, S0c=S0c, S0n=hn["S0"], hydro_rhoY0=hc["rhoY0"],
                strat_inv=np.ones(grid.elem_sc[1]), rhs_out=np.zeros(grid.node_isc), scratch=np.zeros(grid.node_isc))
    gi, gd = _geom(grid, prm, dt, wind)
    lib = _lib.load()
    for part in ("xp", "fw"):
        F = [np.ascontiguousarray(Sol[k]).copy() for k in FIELDS]
        ph, rhs, dp = p2.copy(), np.zeros(grid.node_isc), np.zeros(grid.node_isc)
        fp = (ctypes.c_void_p * 6)(*[a.ctypes.data for a in F])
        tail = (_ptr(np.ascontiguousarray(hn["S0"])), _ptr(np.ascontiguousarray(hc["rhoY0"])),
                _ptr(base["strat_inv"]))
        keep = _dev(base)
        a = _args(_lib.Expl3D, grid, prm, dt, keep)
        for q in range(3):
            a.wind[q] = wind[q]
        if part == "xp":
            host_lib.e3_host_expl_part(_ptr(gi), _ptr(gd), fp, *tail)
            assert lib.bella_expl_part3d(ctypes.byref(a), None) == 0
        else:
            host_lib.e3_host_forward(_ptr(gi), _ptr(gd), fp, _ptr(ph), _ptr(rhs), _ptr(dp), _ptr(S0c), *tail)
            assert lib.bella_euler_forward3d(ctypes.byref(a), None) == 0
        torch.cuda.synchronize()
        for k, h in zip(FIELDS, F):
            _close(keep[k], h, what=(part, k))
        if part == "fw":
            _close(keep["p2"], ph, what="p2")
            mom = max(np.abs(Sol[k]).max() for k in ("rhou", "rhov", "rhow"))
            _close(keep["rhs_out"], rhs, mom / min(grid.dx, grid.dy, grid.dz), "rhs")


@pytest.mark.parametrize("regime", ["plain", "cor"])
@pytest.mark.parametrize("shape", SHAPES)
def test_implicit_pieces_match_the_oracle(shape, regime):
    import torch
    from oracle import nodal3d as n3, proj3d as o3
    from pybella_gb300 import _lib
    grid, prm, Sol, p2, hn, hc, sf, _ = _inputs(shape, regime, seed=9)
    dt = 0.02
    ops = []

    def none(op, b, tol, maxiter):
        ops.append(op)
        return np.zeros_like(b), 1, 0

    So, po = {k: v.copy() for k, v in Sol.items()}, p2.copy()
    out = o3.impl_part(So, po, hn["S0"], hc, sf, grid, prm, dt, solver=none)
    keep = _dev(dict({k: Sol[k] for k in FIELDS}, p2=p2, S0n=hn["S0"], hydro_rhoY0=hc["rhoY0"],
                     strat_inv=np.ones(grid.elem_sc[1]), rhs_out=np.zeros(grid.node_isc)))
    a = _args(_lib.Proj3D, grid, prm, dt, keep)
    a.precond = 0
    ws, o, st = _lib.Workspace(0), _lib.SolveOpts(), _lib.SolveStats()
    ws._lib.bella_solve_opts_default(ctypes.byref(o))
    o.maxiter, o.precision, o.tol = 0, 0, 1e-12
    rc = ws._lib.bella_projection3d(ws.handle, ctypes.byref(a), ctypes.byref(o), ctypes.byref(st), None)
    assert rc >= 0 and st.iterations == 0
    torch.cuda.synchronize()
    mom = max(np.abs(Sol[k]).max() for k in ("rhou", "rhov", "rhow"))
    _close(keep["rhs_out"], out["rhs"], mom / (min(grid.dx, grid.dy, grid.dz) * dt), "rhs")
    for k in FIELDS:
        _close(keep[k], So[k], what=k)
    _close(keep["p2"], po, what="p2")
    x = np.random.default_rng(8).standard_normal(grid.inx * grid.iny * grid.inz)
    dx = torch.tensor(x, device="cuda")
    dy = torch.empty_like(dx)
    assert ws._lib.bella_apply_f64(ws.handle, ctypes.c_void_p(dx.data_ptr()), ctypes.c_void_p(dy.data_ptr()), None) == 0
    torch.cuda.synchronize()
    _close(dy, n3.lap3d(x, ops[0]), what="operator")
