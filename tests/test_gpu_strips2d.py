"""The strips of the 2D operator and the whole-iteration launch at their edges: grids narrower and
wider than a strip (30 columns, double-float 62) and its multiples, heights below a strip's, odd
node counts, an unaligned solution vector, with and without Coriolis cross terms and
hcenter; one BiCGStab iteration of each precision against scipy's control flow in
NumPy, and against the same iteration in three launches.

Tolerance: the operator within 1e-13 of the oracle's (tests/test_gpu_operator.py); two
iterations amplify the rounding of their sums by the ratios of norms in alpha, beta and
omega, measured below 100 on these systems: 1e-11 FP64 and 1e-10 double-float (4e-15 a
value)."""
import ctypes

import numpy as np
import pytest

from oracle import nodal2d as n2

pytestmark = pytest.mark.gpu

SIZES = [(3, 3), (5, 40), (29, 7), (30, 8), (31, 9), (61, 5), (62, 66), (63, 33), (125, 64), (157, 129), (400, 3)]


def _op(nx, ny, cross, hc, seed=3):
    rng = np.random.default_rng(seed)
    nc, n = (nx + 1) * (ny + 1), nx * ny
    pos = lambda m: 0.5 + rng.random(m)
    hx = pos(nc)
    cor = (pos(nc), pos(nc), 0.3 * rng.standard_normal(nc) if cross else np.zeros(nc),
           0.3 * rng.standard_normal(nc) if cross else np.zeros(nc))
    h = -5.0 * pos(n) if hc else np.zeros(n)
    dx, dy = 0.1, 0.13
    return dict(hplusx=hx, hplusy=hx.copy(), hcenter=h, cor=cor, diag_inv=-pos(n) / (4.0 / dx ** 2), nx=nx, ny=ny,
                dx=dx, dy=dy, x_wall=False, y_wall=True)


def _dev(op, ws=None):
    from pybella_gb300.linalg import NodalHelmholtz2D
    return NodalHelmholtz2D(op["hplusx"], op["hplusy"], op["hcenter"], op["cor"], op["diag_inv"], op["nx"], op["ny"],
                            op["dx"], op["dy"], op["x_wall"], op["y_wall"], ws=ws)


def _bicgstab(op, b, iters):
    """scipy's bicgstab from x = 0, exactly ``iters`` iterations."""
    x, r = np.zeros_like(b), b.copy()
    rh, p, v, rho, alpha, omega = r.copy(), None, None, r @ r, 1.0, 1.0
    prev = rho
    for k in range(iters):
        p = r.copy() if k == 0 else r + (rho / prev) * (alpha / omega) * (p - omega * v)
        v = n2.lap2d_gather(p, op)
        alpha = rho / (rh @ v)
        s = r - alpha * v
        t = n2.lap2d_gather(s, op)
        omega = (t @ s) / (t @ t)
        x = x + alpha * p + omega * s
        r = s - omega * t
        prev, rho = rho, rh @ r
    return x


@pytest.mark.parametrize("cross,hc", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_operator_and_iterations(nx, ny, cross, hc):
    import torch
    op = _op(nx, ny, cross, hc)
    A = _dev(op)
    rng = np.random.default_rng(4)
    p = rng.standard_normal(A.n)
    ref = n2.lap2d_gather(p, op)
    assert np.abs(A.matvec(p) - ref).max() <= 1e-13 * np.abs(ref).max()
    b = n2.lap2d_gather(rng.standard_normal(A.n), op)
    for prec, tol in (("fp64", 1e-11), ("df64", 1e-10)):
        for iters in (1, 2):
            want = _bicgstab(op, b, iters)
            x, st = A.solve(b, tol=1e-300, maxiter=iters, precision=prec)
            assert st["iterations"] == iters
            err = np.abs(x.cpu().numpy() - want).max() / np.abs(want).max()
            assert err <= tol, (prec, iters, err)
            A.ws.profile(True)                 # a kernel per phase
            y, _ = A.solve(b, tol=1e-300, maxiter=iters, precision=prec)
            A.ws.profile(False)
            assert float((x - y).abs().max()) <= tol * np.abs(want).max()
    buf = torch.zeros(A.n + 1, dtype=torch.float64, device="cuda")
    assert buf.data_ptr() % 16 == 0
    z, _ = A.solve(b, tol=1e-300, maxiter=2, out=buf[1:])          # 8 bytes off a 16-byte boundary
    x, _ = A.solve(b, tol=1e-300, maxiter=2)
    assert torch.equal(z, x)


def test_state_and_limits():
    """The stop tests of a launch of many iterations are those of single ones: the iteration limit, the
    tolerance, a zero right-hand side and one that is not finite."""
    from pybella_gb300 import _lib
    op = _op(61, 33, False, True)
    A = _dev(op)
    b = n2.lap2d_gather(np.random.default_rng(5).standard_normal(A.n), op)
    for prec in ("fp64", "df64"):
        for m in (1, 15, 16, 17):
            _, st = A.solve(b, tol=1e-300, maxiter=m, precision=prec)
            assert st["status"] == _lib.BELLA_MAXITER and st["iterations"] == m
        _, st = A.solve(b, tol=1e-9, maxiter=2000, precision=prec, check_every=1)
        _, s2 = A.solve(b, tol=1e-9, maxiter=2000, precision=prec)
        assert st["status"] == s2["status"] == _lib.BELLA_OK and st["iterations"] == s2["iterations"]
        assert st["relres"] <= 1e-9
        x, st = A.solve(np.zeros_like(b), precision=prec)
        assert st["status"] == _lib.BELLA_OK and not x.any()
        bad = b.copy()
        bad[7] = np.nan
        assert A.solve(bad, precision=prec)[1]["status"] == _lib.BELLA_NONFINITE
