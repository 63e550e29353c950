"""The 2D background solve on cells hundreds of times as high as wide, singular and regular: what FP32
transforms leave there is beyond the rounding of the solution itself, which
test_gpu_lines2d.py's tolerance is made of.

Tolerance: that one, and three times what the FP64 oracle's own apply leaves when each transform's
values get one FP32 rounding per butterfly stage, relative to the line's RMS (the rounding of an
FFT spreads over its line): the largest of three draws."""
import numpy as np
import pytest

from oracle import cases, nodal2d as n2, spectral2d
from test_gpu_lines2d import _apply, _seam

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("compressible", [False, True])
@pytest.mark.parametrize("nx,ny", [(2049, 5), (1025, 4), (2049, 9)])
def test_apply2d_on_tall_cells(nx, ny, compressible):
    op = cases.stratified_2d(3, nx, ny, compressible=compressible)["op"]
    ref = spectral2d.BackgroundInverse2D(op)
    r = n2.lap2d_gather(_seam(np.random.default_rng(6), nx, ny), op).astype(np.float32).astype(np.float64)
    y_ref = ref.apply(r)
    res = lambda v: np.linalg.norm(n2.lap2d_gather(v, op))
    R = (r * ref.D).reshape(ref.shape)
    stages = np.sqrt(np.ceil(np.log2(nx)))
    model = []
    for seed in range(3):
        rng = np.random.default_rng(seed)

        def rounded(z):
            e = 2.0 ** -24 * stages * np.sqrt((np.abs(z) ** 2).mean(axis=1, keepdims=True))
            d = rng.uniform(-1.0, 1.0, z.shape)
            return z + e * (d + 1j * rng.uniform(-1.0, 1.0, z.shape) if np.iscomplexobj(z) else d)

        X = np.einsum("kab,bk->ak", ref.Kinv, rounded(ref.fx(R.astype(complex), 1)))
        model.append(res(rounded(np.real(ref.ix(X, 1))).reshape(-1) - y_ref))
    floor = res(y_ref.astype(np.float32).astype(np.float64) - y_ref)
    err = res(_apply(op, r) - y_ref)
    assert err <= 20.0 * floor + 1e-6 * np.linalg.norm(r) + 3.0 * max(model), (err, floor, model)
