"""The ensemble launch at the edges of its strips and runs: members from one strip to several blocks,
with and without cross terms and hcenter mixed in one launch, more members than warps, more
members in a block than it has room for in shared memory, an unaligned solution, members that stop
at once.  Oracle and tolerance as in test_gpu_strips2d.py."""
import numpy as np
import pytest

from test_gpu_strips2d import _bicgstab, _dev, _op

pytestmark = pytest.mark.gpu

SIZES = [(3, 3), (63, 64), (30, 7), (200, 150), (31, 5), (3, 90), (125, 33), (301, 65), (62, 2), (5, 5)]


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("df64", 1e-10)])
@pytest.mark.parametrize("config", [0, 5])
@pytest.mark.parametrize("copies", [1, 30])
def test_mixed_members(precision, tol, config, copies):
    import torch
    from pybella_gb300 import ensemble
    sizes = [(nx, max(ny, 3)) for nx, ny in SIZES]
    ops = [_op(nx, ny, k % 3 == 1, k % 2 == 0, seed=k) for k, (nx, ny) in enumerate(sizes)]
    bs = [np.random.default_rng(50 + k).standard_normal(op["nx"] * op["ny"]) for k, op in enumerate(ops)]
    want = [_bicgstab(op, b, 2) for op, b in zip(ops, bs)]
    dev = [_dev(op) for _ in range(copies) for op in ops]
    out = [torch.zeros(A.n + 1, dtype=torch.float64, device="cuda")[k % 2:][:A.n] for k, A in enumerate(dev)]
    bd = [torch.as_tensor(b, device="cuda") for b in bs] * copies
    xs, st = ensemble.solve_ensemble(dev, bd, tol=1e-300, maxiter=2, config=config, out=out, precision=precision)
    for k, (x, s) in enumerate(zip(xs, st)):
        w = want[k % len(want)]
        assert s["iterations"] == 2 and s["status"] == 1
        assert np.abs(x.cpu().numpy() - w).max() <= tol * np.abs(w).max(), k
        r = torch.linalg.norm(bd[k] - dev[k].matvec(x)) / torch.linalg.norm(bd[k])
        assert abs(float(r) - s["relres"]) <= 1e-9 * float(r)


@pytest.mark.parametrize("precision", ["fp64", "df64"])
def test_members_that_stop_at_once(precision):
    import torch
    from pybella_gb300 import _lib, ensemble
    op = _op(63, 64, False, True)
    dev = [_dev(op) for _ in range(4)]
    b = torch.as_tensor(np.random.default_rng(1).standard_normal(63 * 64), device="cuda")
    bad = b.clone()
    bad[11] = float("inf")
    xs, st = ensemble.solve_ensemble(dev, [b, torch.zeros_like(b), bad, 1e-30 * b], tol=1e-10, maxiter=3, config=0,
                                     precision=precision)
    # ||b|| <= tol stops with x = 0; double-float members then are refined to tol ||b||
    small = precision == "fp64"
    assert [s["status"] for s in st] == [_lib.BELLA_MAXITER, _lib.BELLA_OK, _lib.BELLA_NONFINITE,
                                         _lib.BELLA_OK if small else _lib.BELLA_MAXITER]
    assert [s["iterations"] for s in st] == [3, 0, 0, 0 if small else 3]
    assert not xs[1].any() and not xs[2].any() and bool(torch.isfinite(xs[0]).all())
    assert bool(xs[3].any()) != small
    # no iteration allowed
    xs, st = ensemble.solve_ensemble(dev[:1], [b], tol=1e-10, maxiter=0, config=0, precision=precision)
    assert st[0]["status"] == _lib.BELLA_MAXITER and st[0]["iterations"] == 0 and not xs[0].any()


def test_more_members_than_a_block_holds():
    import torch
    from pybella_gb300 import ensemble
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    op = _op(4, 3, False, True)
    b = np.random.default_rng(2).standard_normal(12)
    want = _bicgstab(op, b, 2)
    A = [_dev(op) for _ in range(33 * sms + 5)]
    bd = torch.as_tensor(b, device="cuda")
    xs, st = ensemble.solve_ensemble(A, [bd] * len(A), tol=1e-300, maxiter=2, config=0)
    got = torch.stack(xs).cpu().numpy()
    assert np.abs(got - want).max() <= 1e-10 * np.abs(want).max()
