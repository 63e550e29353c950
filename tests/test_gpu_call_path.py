"""Calls into the library from other streams and with other kinds of vectors than the usual ones."""
import numpy as np
import pytest

from test_gpu_strips2d import _dev, _op

pytestmark = pytest.mark.gpu


def test_vectors_and_streams():
    import torch
    op = _op(63, 40, True, True)
    A = _dev(op)
    p = torch.as_tensor(np.random.default_rng(0).standard_normal(A.n), device="cuda")
    want = A.matvec(p)
    wide = torch.empty(A.n, 2, dtype=torch.float64, device="cuda")
    wide[:, 0] = p
    forms = [p.reshape(40, 63), wide[:, 0], p.clone().requires_grad_(), torch.nn.Parameter(p.clone()), p.cpu(),
             p.cpu().numpy(), p.cpu().numpy()[::-1].copy()[::-1]]
    for q in forms:
        y = A.matvec(q)
        y = torch.as_tensor(y, device="cuda")
        assert torch.equal(y, want) and not y.requires_grad
    assert torch.equal(A.matvec(p.float()), A.matvec(p.float().double()))
    with pytest.raises(ValueError):
        A.matvec(p[:-1])
    # on another stream: ordered with that stream's work
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(2_000_000)
        q = 2.0 * p
        y = A.matvec(q)
        x, st = A.solve(q, tol=1e-300, maxiter=3)
    side.synchronize()
    assert torch.allclose(y, 2.0 * want, rtol=1e-15, atol=0.0)
    assert torch.equal(x, A.solve(2.0 * p, tol=1e-300, maxiter=3)[0])
    # the caller's vector is not the result, nor changed
    assert A.matvec(p).data_ptr() != p.data_ptr()
    b = p.clone()
    A.solve(b, tol=1e-300, maxiter=3)
    assert torch.equal(b, p)
