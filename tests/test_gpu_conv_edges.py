"""The convolution's and the weight gradients' staging at its edges: planes of one short line after the
other, lines about as long as fit, shares that cross from one row block to the next (the rows
outside the plane change), one voxel more or less than a row block.  Against the mma.sync and
CUDA-core kernels; tolerances of test_gpu_cnn.py (the same BF16 operands, FP32 sums in another order)."""
import numpy as np
import pytest

from test_gpu_cnn import _params, _rel

pytestmark = pytest.mark.gpu

SHAPES = [(1, (5, 3, 3)), (1, (4, 200, 3)), (2, (9, 5, 262)), (1, (121, 30, 30)), (2, (7, 28, 28)), (1, (3, 14, 15)),
          (1, (2, 62, 2))]


@pytest.mark.parametrize("block,shape", SHAPES)
def test_against_the_other_kernels(block, shape):
    import torch
    from pybella_gb300.learned import CNN
    rng = np.random.default_rng(sum(shape))
    params = _params(block, 9)
    for l in range(6):
        params["b%d" % l] = np.zeros_like(params["b%d" % l])
    n = int(np.prod(shape))
    x = torch.tensor(rng.standard_normal(n), dtype=torch.float32, device="cuda")
    gout = torch.tensor(rng.standard_normal(n), dtype=torch.float32, device="cuda")
    net = CNN(shape, block=block, mode="linear")
    net.set_params(params)
    y, g = {}, {}
    for tc in (False, True):
        net.set_tensor_cores(tc)
        y[tc] = net.forward(x, shape, scale=1.0).cpu().numpy()
        g[tc] = net.gradients(x, gout, shape)[0].cpu().numpy()
    assert not net.tensor_core_error()
    assert _rel(y[True], y[False]) < 1e-2
    assert _rel(g[True], g[False]) < 1e-2
    z = net.forward(x, shape, scale=1.0).cpu().numpy()              # the same again
    assert np.array_equal(y[True], z)
