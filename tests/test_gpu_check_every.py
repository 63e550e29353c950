"""check_every is in force: a plain 2D FP64 solve takes a launch for each block of that many iterations, a solve
with the network as preconditioner looks every one to four, and the results do not depend on it."""
import numpy as np
import pytest

from test_gpu_strips2d import _dev, _op

pytestmark = pytest.mark.gpu


def test_plain_2d():
    import torch
    A = _dev(_op(61, 33, False, True))
    b = torch.as_tensor(np.random.default_rng(5).standard_normal(A.n), device="cuda")

    def run(**kw):
        l0 = A.ws.launches
        x, st = A.solve(b, tol=1e-300, maxiter=24, precision="fp64", **kw)
        assert st["iterations"] == 24
        return x, A.ws.launches - l0

    x1, l1 = run(check_every=1)
    x8, l8 = run(check_every=8)
    x24, l24 = run(check_every=24)
    x, _ = run()
    assert (l1 - l24, l8 - l24) == (23, 2)
    assert all(torch.equal(x, y) for y in (x1, x8, x24))


def test_network_as_preconditioner():
    import torch
    from pybella_gb300 import learned, workloads
    shape = (33, 17, 33)
    w = workloads.stratified_3d(1, *shape)
    A = learned.operator_3d(w)
    net = learned.CNN(shape, block=2, mode="linear", skip=0.9)
    net.init(3, last_gain=0.1)

    def run(**kw):
        l0 = A.ws.launches
        x, st = A.solve(w["b"], tol=1e-3, maxiter=5, max_outer=1, preconditioner=net, **kw)
        return x, A.ws.launches - l0

    (x1, l1), (x2, l2), (x4, l4) = run(check_every=1), run(check_every=2), run()
    assert torch.equal(x1, x2) and torch.equal(x1, x4)
    assert l1 < l2 < l4            # an inner solve that ends inside a block launches the block's rest
