"""Domains whose tiles along one axis pass 65,535, the largest y and z extent of a launch's grid: the
advection in 2D and 3D and the 3D projection's explicit parts.  All axes are periodic, without gravity,
and the data repeat every PERIOD cells of the long axis, so the result is that of a domain of one
period (of which other tests hold the values) repeated.

Tolerance: both sides evaluate the same formulas, their sums perhaps in another order: 1e-12 of the
maximum as in test_gpu_sweeps.py, the divergence of its momenta over the spacing."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PERIOD = 64
LONG = 4 + PERIOD * (8 * 65536 // PERIOD)
FIELDS = ("rho", "rhou", "rhov", "rhow", "rhoY", "rhoX")


def _fields(n, axis, extra, seed):
    """The fields on n cells (n - 4 of them within a period) plus ``extra`` along every axis."""
    import torch
    rng = np.random.default_rng(seed)
    period = [PERIOD if d == axis else n[d] - 4 for d in range(len(n))]
    rho = 1.0 + 0.1 * rng.random(period)
    base = [rho] + [0.1 * rng.standard_normal(period) for _ in range(3)] + [1.0 + 0.1 * rng.random(period),
                                                                          0.1 * rng.standard_normal(period)]
    out = []
    for t in base:
        t = torch.tensor(t, device="cuda")
        for d, p in enumerate(period):
            t = t.index_select(d, torch.arange(n[d] + extra, device="cuda") % p)
        out.append(t.contiguous())
    return out


def _repeats(long, short, dim, what, scale=None):
    """Entries 3 .. n-4 along ``dim`` of the long array are those of the short one, repeated."""
    import torch
    at = torch.arange(3, long.shape[dim] - 4, device="cuda")
    a, b = long.index_select(dim, at), short.index_select(dim, 3 + (at - 3) % PERIOD)
    s = float(b.abs().max()) if scale is None else scale
    assert float((a - b).abs().max()) <= 1e-12 * s, what


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _advect(n, axis, what):
    import torch
    from pybella_gb300 import _lib
    nd = len(n)
    f = _fields(n, axis, 0, 2)
    a = _lib.Adv3D() if nd == 3 else _lib.Adv2D()
    faces, order = [], []
    for s in range(nd):
        order.append([(s + 1 + q) % nd for q in range(nd)])
        shape = [n[d] + (d == s) for d in order[s]]
        faces.append([torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in FIELDS])
    a.inx, a.iny, a.dx, a.dy, a.gamm = n[0] - 3, n[1] - 3, 0.1, 0.07, 1.4
    if nd == 3:
        a.inz, a.dz = n[2] - 3, 0.13
    for k, t in zip(FIELDS, f):
        setattr(a, k, _p(t))
    for s, nm in enumerate(("fx", "fy", "fz")[:nd]):
        for q in range(6):
            getattr(a, nm)[q] = _p(faces[s][q])
    col = torch.ones(n[1], dtype=torch.float64, device="cuda")
    a.hydro_rhoY0 = a.strat_inv = _p(col)
    lib = _lib.load()
    call = lambda fn, *args: getattr(lib, "bella_%s%dd" % (fn, nd))(ctypes.byref(a), *args, None)
    assert call("boundary") == 0 and call("advective_fluxes") == 0
    assert (call("advect_rk", 0.02) if what == "rk" else call("advect", 0.02, 1)) == 0
    torch.cuda.synchronize()
    return f, [(t[4], o.index(axis)) for t, o in zip(faces, order)]


@pytest.mark.parametrize("what", ["rk", "strang"])
@pytest.mark.parametrize("nd,axis", [(2, 0), (2, 1), (3, 0), (3, 1), (3, 2)])
def test_advection(nd, axis, what):
    n = lambda m: [m if d == axis else 8 for d in range(nd)]
    f, mass = _advect(n(LONG), axis, what)
    f1, mass1 = _advect(n(4 + PERIOD), axis, what)
    for k, a, b in zip(FIELDS, f, f1):
        _repeats(a, b, axis, k)
    for (a, dim), (b, _) in zip(mass, mass1):
        _repeats(a, b, dim, "mass")


def _explicit(n, axis, part):
    import torch
    from pybella_gb300 import _lib
    f = _fields(n, axis, 0, 3)
    nodes = _fields(n, axis, 1, 5)
    isc = [k - 1 for k in n]
    z = lambda shape: torch.zeros(shape, dtype=torch.float64, device="cuda")
    dev = dict(zip(FIELDS, f), p2=nodes[1], S0c=f[0].clone(), rhs_out=z(isc), scratch=z(isc), S0n=1.0 + z(n[1] + 1),
               hydro_rhoY0=1.0 + z(n[1]), strat_inv=1.0 + z(n[1]))
    a = _lib.Expl3D()
    a.inx, a.iny, a.inz = (k - 3 for k in n)
    a.dx = a.dy = a.dz = 0.1
    a.dt, a.Msq, a.gamm, a.nonhydro, a.coriolis[1] = 0.01, 0.1, 1.4, 1.0, 0.5
    for k, t in dev.items():
        setattr(a, k, _p(t))
    assert getattr(_lib.load(), "bella_" + part)(ctypes.byref(a), None) == 0
    torch.cuda.synchronize()
    return dev


@pytest.mark.parametrize("part", ["expl_part3d", "euler_forward3d"])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_explicit_parts(axis, part):
    n = lambda m: [m if d == axis else 8 for d in range(3)]
    long, short = _explicit(n(LONG), axis, part), _explicit(n(4 + PERIOD), axis, part)
    for k in FIELDS + ("p2",):
        _repeats(long[k], short[k], axis, k)
    if part == "euler_forward3d":
        _repeats(long["rhs_out"], short["rhs_out"], axis, "rhs", 1.0 / 0.1)
