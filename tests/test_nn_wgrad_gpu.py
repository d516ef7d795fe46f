"""GPU tests of the tensor-core weight gradient's tiling (nn_wgrad.cuh): columns of 16 x 8 voxels cut
off by the volume's edges, segments of z-planes and the flush of the accumulators, against the
CUDA-core kernel (SULI_WGRAD_CUDA_CORES=1).  Both add the same BF16 products in FP32; the tensor
cores truncate, which over a chain of at most 256 products is 2^-17 of the sum of the products'
sizes, and a block of gradients keeps more than a hundredth of that: 1e-3 of its norm."""
import numpy as np
import pytest

from test_nn_gpu import _layer_slices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 8, 8), (24, 40, 72), (40, 24, 16), (16, 8, 136)])
def test_ragged_columns_and_segments(pkg, monkeypatch, shape):
    torch = pytest.importorskip("torch")
    nx, ny, nz = shape
    rng = np.random.default_rng(17)
    theta = pkg.learned.init_params(17, head_scale=1.0)
    x3 = torch.from_numpy(rng.standard_normal((nx * ny * nz, 3)).astype(np.float32)).to("cuda:0")
    t = torch.from_numpy(rng.standard_normal(nx * ny * nz).astype(np.float32)).to("cuda:0")
    grads = {}
    for cores in ("1", "0"):
        monkeypatch.setenv("SULI_WGRAD_CUDA_CORES", cores)
        net = pkg.learned.Net(nx, ny, nz, params=theta)
        _, g = net.loss_grad(x3, t)
        assert np.array_equal(g, net.loss_grad(x3, t)[1])
        grads[cores] = g.astype(np.float64)
        net.close()
    for name, sl in _layer_slices():
        a, b = grads["0"][sl], grads["1"][sl]
        assert np.linalg.norm(a - b) <= 1e-3 * max(np.linalg.norm(b), 1e-30), name
