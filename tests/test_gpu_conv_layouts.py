"""The network where its paths and the layouts of its activations change: the last z extent whose planes
fit the tcgen05 convolution (142 voxels), those where only the weight gradients' planes do (planes of 8
channels read by the mma.sync convolution), the first where neither does (a voxel's channels
together); linear and with ReLUs, whose masks are read in the same layout.  Against the mma.sync and
CUDA-core kernels as test_gpu_conv_edges.py, whose tolerance this is."""
import numpy as np
import pytest

from test_gpu_cnn import _params, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["linear", "relu"])
@pytest.mark.parametrize("block,nz", [(1, 142), (1, 143), (1, 154), (1, 155), (2, 286), (2, 311)])
def test_against_the_other_kernels(block, nz, mode):
    import torch
    from pybella_gb300.learned import CNN
    shape = (5, 6, nz)
    rng = np.random.default_rng(nz)
    n = int(np.prod(shape))
    x = torch.tensor(rng.standard_normal(n), dtype=torch.float32, device="cuda")
    gout = torch.tensor(rng.standard_normal(n), dtype=torch.float32, device="cuda")
    net = CNN(shape, block=block, mode=mode)
    params = _params(block, 9)
    if mode == "linear":
        for l in range(6):
            params["b%d" % l] = np.zeros_like(params["b%d" % l])
    net.set_params(params)
    y, g = {}, {}
    for tc in (False, True):
        net.set_tensor_cores(tc)
        y[tc] = net.forward(x, shape, scale=1.0).cpu().numpy()
        g[tc] = net.gradients(x, gout, shape)[0].cpu().numpy()
    assert not net.tensor_core_error()
    assert _rel(y[True], y[False]) < 1e-2
    assert _rel(g[True], g[False]) < 1e-2
