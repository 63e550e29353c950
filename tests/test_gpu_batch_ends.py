"""What an ensemble's solve leaves in x for members that end not finite: x0 = 0 where the
right-hand side is not finite, the last iterate where the iteration overflows after some steps; the same
with the caller's vectors and with the solve's own, in both precisions."""
import numpy as np
import pytest

from test_gpu_strips2d import _dev, _op

pytestmark = pytest.mark.gpu


def _overflowing():
    """A member whose right-hand side lies to the left of coefficients of 1e30: the iteration reaches
    them after a few steps, and its inner products leave FP32's range."""
    op = _op(201, 5, False, True)
    h = op["hplusx"].reshape(6, 202)
    h[:, 60:140] *= 1e30
    op["hplusy"] = op["hplusx"].copy()
    b = np.zeros((5, 201))
    b[:, 20:40] = np.random.default_rng(3).standard_normal((5, 20))
    return op, b.reshape(-1)


@pytest.mark.parametrize("precision", ["fp64", "df64"])
def test_x_of_members_that_end_not_finite(precision):
    import torch
    from pybella_gb300 import _lib, ensemble
    good = _op(63, 64, False, True)
    over, bo = _overflowing()
    b = np.random.default_rng(1).standard_normal(63 * 64)
    bad = b.copy()
    bad[11] = np.inf
    dev = [_dev(good), _dev(good), _dev(over)]
    bs = [torch.as_tensor(v, device="cuda") for v in (b, bad, bo)]
    kw = dict(tol=1e-10, maxiter=40, config=0, precision=precision)
    xs, st = ensemble.solve_ensemble(dev, bs, **kw)
    own = [torch.full_like(v, 7.0) for v in bs]
    ys, s2 = ensemble.solve_ensemble(dev, bs, out=own, **kw)
    assert [s["status"] for s in st] == [s["status"] for s in s2]
    for x, y in zip(xs, ys):
        assert torch.equal(x, y)
    assert st[1]["status"] == _lib.BELLA_NONFINITE and not xs[1].any()
    if precision == "df64":
        assert st[2]["status"] == _lib.BELLA_NONFINITE and st[2]["iterations"] > 0
        assert bool(xs[2].any()) and bool(torch.isfinite(xs[2]).all())
