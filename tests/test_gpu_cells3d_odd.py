"""Cells that are not finite, or zero, in the 3D projection's cell and node kernels: a NaN, an infinity or a
zero in one field of one cell (or in one node of the pressure) reaches the values that it reaches in
the host build of bella_expl3d.cuh and in the oracle's implicit part; what stays finite agrees as in
test_gpu_cells3d.py, whose tolerance this is."""
import ctypes

import numpy as np
import pytest

from test_expl3d_host import FIELDS, _geom, _ptr, host_lib  # noqa: F401
from test_gpu_cells3d import _args, _dev, _inputs

pytestmark = pytest.mark.gpu

SHAPE = (13, 9, 11)
CELL = (7, 6, 5)


def _same(got, ref, what, scale=None):
    got = got.cpu().numpy()
    ok = np.isfinite(ref)
    assert np.array_equal(ok, np.isfinite(got)), (what, int((ok != np.isfinite(got)).sum()))
    s = np.abs(ref[ok]).max() if scale is None else scale
    assert np.abs(got[ok] - ref[ok]).max() <= 1e-12 * max(s, 1e-300), what


@pytest.mark.parametrize("bad", [np.nan, np.inf, 0.0])
@pytest.mark.parametrize("q", FIELDS + ("p2",))
@pytest.mark.parametrize("regime", ["plain", "cor"])
def test_explicit_parts_keep_what_is_not_finite(host_lib, regime, q, bad):  # noqa: F811
    import torch
    from pybella_gb300 import _lib
    grid, prm, Sol, p2, hn, hc, sf, wind = _inputs(SHAPE, regime)
    (p2 if q == "p2" else Sol[q])[CELL] = bad
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
        for k in range(3):
            a.wind[k] = wind[k]
        if part == "xp":
            host_lib.e3_host_expl_part(_ptr(gi), _ptr(gd), fp, *tail)
            assert lib.bella_expl_part3d(ctypes.byref(a), None) == 0
        else:
            host_lib.e3_host_forward(_ptr(gi), _ptr(gd), fp, _ptr(ph), _ptr(rhs), _ptr(dp), _ptr(S0c), *tail)
            assert lib.bella_euler_forward3d(ctypes.byref(a), None) == 0
        torch.cuda.synchronize()
        for k, h in zip(FIELDS, F):
            _same(keep[k], h, (part, k))
        if part == "fw":
            _same(keep["p2"], ph, "p2")
            mom = max(np.nanmax(np.where(np.isfinite(Sol[k]), np.abs(Sol[k]), 0.0)) for k in ("rhou", "rhov", "rhow"))
            _same(keep["rhs_out"], rhs, "rhs", mom / min(grid.dx, grid.dy, grid.dz))


@pytest.mark.parametrize("bad", [np.nan, np.inf, 0.0])
@pytest.mark.parametrize("q", FIELDS + ("p2",))
@pytest.mark.parametrize("regime", ["plain", "cor"])
def test_correction_keeps_what_is_not_finite(regime, q, bad):
    """The implicit part, its solve stopped before the first iteration."""
    import torch
    from oracle import proj3d as o3
    from pybella_gb300 import _lib
    grid, prm, Sol, p2, hn, hc, sf, _ = _inputs(SHAPE, regime, seed=9)
    (p2 if q == "p2" else Sol[q])[CELL] = bad
    dt = 0.02
    So, po = {k: v.copy() for k, v in Sol.items()}, p2.copy()
    with np.errstate(all="ignore"):
        o3.impl_part(So, po, hn["S0"], hc, sf, grid, prm, dt, solver=lambda op, b, tol, maxiter: (np.zeros_like(b), 1, 0))
    keep = _dev(dict({k: Sol[k] for k in FIELDS}, p2=p2, S0n=hn["S0"], hydro_rhoY0=hc["rhoY0"],
                     strat_inv=np.ones(grid.elem_sc[1])))
    a = _args(_lib.Proj3D, grid, prm, dt, keep)
    a.precond = 0
    ws, o, st = _lib.Workspace(0), _lib.SolveOpts(), _lib.SolveStats()
    ws._lib.bella_solve_opts_default(ctypes.byref(o))
    o.maxiter, o.precision, o.tol = 0, 0, 1e-12
    assert ws._lib.bella_projection3d(ws.handle, ctypes.byref(a), ctypes.byref(o), ctypes.byref(st), None) >= 0
    torch.cuda.synchronize()
    for k in FIELDS:
        _same(keep[k], So[k], k)
    _same(keep["p2"], po, "p2")
