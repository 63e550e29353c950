"""The launch of whole BiCGStab iterations in each of its layouts: a block for four, two or one of the full
layout's blocks, one with two shares of the vector update a warp, and a block an SM.  Against a kernel a
phase, whose sums have another order; tolerances of test_gpu_strips2d.py.  An unaligned solution takes
other loads and gives the same bits."""
import numpy as np
import pytest

from test_gpu_strips2d import _dev, _op

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("df64", 1e-10)])
@pytest.mark.parametrize("cross,hc", [(False, True), (True, False)])
@pytest.mark.parametrize("nx,ny", [(65, 33), (160, 81), (225, 113), (448, 225), (641, 321), (1600, 1100)])
def test_layouts(nx, ny, cross, hc, precision, tol):
    import torch
    A = _dev(_op(nx, ny, cross, hc))
    b = A.matvec(torch.as_tensor(np.random.default_rng(4).standard_normal(A.n), device="cuda"))
    kw = dict(tol=1e-300, maxiter=2, precision=precision)
    x, st = A.solve(b, **kw)
    assert st["iterations"] == 2
    A.ws.profile(True)
    y, _ = A.solve(b, **kw)
    A.ws.profile(False)
    assert float((x - y).abs().max()) <= tol * float(y.abs().max())
    z, _ = A.solve(b, out=torch.zeros(A.n + 1, dtype=torch.float64, device="cuda")[1:], **kw)
    assert torch.equal(z, x)
    x1, _ = A.solve(b, check_every=1, **kw)
    assert torch.equal(x1, x)
