"""The line sweeps and mass-flux planes of bella_advect.cu at the edges of their tiles,
against the host build of bella_advect.cuh (tests/advect_host.cpp): every block
shape (1, 4 or 32 lines, 8 contiguous ones), lines shorter and longer than a block's
chunk, remainders of every tile, walls and periodic axes, gravity on and off, the
compressible reflection, and cells that are not finite.

Tolerance: a cell's result is a sum of terms no larger than the field's maximum, each
from fewer than 100 FP64 operations (100 eps = 2e-14 of it) in each of at most eight
passes, so 1e-12 of the field's maximum leaves a factor of six; pow in the
compressible reflection adds a few ulp."""
import ctypes

import numpy as np
import pytest

from test_advect_host import FIELDS, _ptrs, host_lib  # noqa: F401

pytestmark = pytest.mark.gpu

# (cells incl. ghosts, walls): lines per block follow from the line counts
CASES = [((8, 8), (0, 1)), ((41, 74), (1, 1)), ((11, 1303), (0, 0)), ((300, 9), (0, 1)), ((2500, 8), (1, 1)),
         ((8, 8, 8), (0, 1, 0)), ((15, 12, 43), (1, 1, 1)), ((24, 43, 41), (0, 0, 1)), ((9, 100, 101), (0, 1, 0)),
         ((105, 25, 9), (1, 1, 0)), ((10, 70, 33), (0, 1, 1)), ((70, 11, 300), (0, 1, 0))]


def _state(ic, seed):
    rng = np.random.default_rng(seed)
    rho = 1.0 + 0.2 * rng.random(ic)
    f = [rho] + [rho * (0.3 * rng.standard_normal(ic)) for _ in range(3)] + [rho * (1.0 + 0.1 * rng.random(ic)),
                                                                            rho * 0.1 * rng.standard_normal(ic)]
    return [np.ascontiguousarray(a) for a in f]


def _both(host, ic, walls, what, comp=0, g=0.9, seed=1, spoil=None):
    """(device arrays, host arrays): the fields, the face arrays and pwchi after the mass fluxes and ``what``."""
    import torch
    from pybella_gb300 import _lib
    nd = len(ic)
    F = _state(ic, seed)
    if spoil:
        spoil(F)
    shapes = ([(ic[1], ic[0] + 1), (ic[0], ic[1] + 1)] if nd == 2 else
              [(ic[1], ic[2], ic[0] + 1), (ic[2], ic[0], ic[1] + 1), (ic[0], ic[1], ic[2] + 1)])
    d = [0.1, 0.07, 0.13][:nd] + [1.0] * (3 - nd)
    rhoY0, sinv = 1.0 + 0.1 * np.cos(np.arange(ic[1])), 1.0 + 0.05 * np.sin(np.arange(ic[1]))
    dt = 0.04
    dF = [torch.tensor(a, device="cuda") for a in F]
    dfaces = [torch.zeros(s, dtype=torch.float64, device="cuda") for s in shapes for _ in FIELDS]
    dpw = torch.zeros(ic, dtype=torch.float64, device="cuda")
    cols = [torch.tensor(a, device="cuda") for a in (rhoY0, sinv)]
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    a = _lib.Adv3D() if nd == 3 else _lib.Adv2D()
    a.inx, a.iny, a.x_wall, a.y_wall = ic[0] - 3, ic[1] - 3, walls[0], walls[1]
    a.dx, a.dy, a.g, a.gamm, a.is_compressible = d[0], d[1], g, 1.4, comp
    if nd == 3:
        a.inz, a.z_wall, a.dz = ic[2] - 3, walls[2], d[2]
    for k, t in zip(FIELDS, dF):
        setattr(a, k, p(t))
    for s, nm in enumerate(("fx", "fy", "fz")[:nd]):
        for q in range(6):
            getattr(a, nm)[q] = p(dfaces[6 * s + q])
    a.hydro_rhoY0, a.strat_inv, a.pwchi = p(cols[0]), p(cols[1]), p(dpw)
    lib, n = _lib.load(), "%dd" % nd
    assert getattr(lib, "bella_advective_fluxes" + n)(ctypes.byref(a), None) == 0
    if what == "rk":
        assert getattr(lib, "bella_advect_rk" + n)(ctypes.byref(a), dt, None) == 0
    else:
        assert getattr(lib, "bella_advect" + n)(ctypes.byref(a), dt, int(what == "odd"), None) == 0
    torch.cuda.synchronize()
    dev = [t.cpu().numpy() for t in dF + dfaces + [dpw]]

    geo = np.array([nd] + list(ic) + [1] * (3 - nd) + list(walls) + [0] * (3 - nd), dtype=np.int32)
    dg = np.array(d + [g, 1.4])
    H = [b.copy() for b in F]
    faces, pw = [np.zeros(s) for s in shapes for _ in FIELDS], np.zeros(ic)
    v = lambda b: ctypes.c_void_p(b.ctypes.data)
    with np.errstate(all="ignore"):
        host.adv_host_mass(v(geo), v(dg), _ptrs(H), _ptrs(faces))
        args = (v(geo), v(dg), ctypes.c_int(comp), _ptrs(H), _ptrs(faces), v(rhoY0), v(sinv))
        if what == "rk":
            host.adv_host_rk(*args, ctypes.c_double(dt), v(pw))
        else:
            host.adv_host_strang(*args, ctypes.c_double(dt), ctypes.c_int(int(what == "odd")))
    return dev, H + faces + [pw]


def _check(dev, host):
    for k, (a, b) in enumerate(zip(dev, host)):
        ok = np.isfinite(b)
        assert np.array_equal(ok, np.isfinite(a)), k
        if ok.any():
            assert np.abs(a[ok] - b[ok]).max() <= 1e-12 * max(np.abs(b[ok]).max(), 1e-300), k


@pytest.mark.parametrize("what", ["odd", "even", "rk"])
@pytest.mark.parametrize("ic,walls", CASES)
def test_sweeps_match_the_host_build(host_lib, ic, walls, what):  # noqa: F811
    _check(*_both(host_lib, ic, walls, what))


@pytest.mark.parametrize("ic,walls", [((41, 74), (0, 1)), ((15, 12, 43), (0, 1, 0))])
def test_sweeps_compressible_and_without_gravity(host_lib, ic, walls):  # noqa: F811
    _check(*_both(host_lib, ic, walls, "odd", comp=1))
    _check(*_both(host_lib, ic, walls, "even", g=0.0))
    _check(*_both(host_lib, ic, walls, "rk", comp=1))


@pytest.mark.parametrize("q", range(6))
@pytest.mark.parametrize("bad", [np.nan, np.inf, 0.0])
def test_sweeps_keep_what_is_not_finite(host_lib, q, bad):  # noqa: F811
    """A NaN, an infinity or a zero in one cell reaches the cells that it reaches on the host."""
    def spoil(F):
        F[q][20, 30] = bad
    for what in ("odd", "rk"):
        _check(*_both(host_lib, (41, 74), (0, 1), what, spoil=spoil))
