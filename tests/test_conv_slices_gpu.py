"""The convolution kernel takes 1 to 8 slices of a volume per block, by how many blocks the
volume gives; every output is the same sum in the same order either way.  So a window's
prediction must be the same bits alone and in a batch, for windows whose padded sizes end
inside a block's 8 x 16 x (1..8) voxels.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(64, 64, 64, 10), (40, 33, 17, 12), (16, 16, 16, 40), (72, 24, 40, 9), (8, 9, 2, 3)], ids=str)
def test_prediction_does_not_depend_on_the_batch(tomo, shape):
    import torch

    nx, ny, nz, n = shape
    h, rng = 10.0, np.random.default_rng(nx)
    slow = torch.from_numpy(rng.uniform(2e-4, 6e-4, (n * ny, nx, nz)).astype(np.float32)).cuda()
    size = nx * ny * nz
    net = tomo.Net(seed=3)

    def predict(which):
        out = torch.full((len(which) * size,), -7.0, dtype=torch.float32, device="cuda")
        net.predict([dict(slow=slow.data_ptr(), model_nx=nx, model_ny=n * ny, nz=nz, window=(0, nx, k * ny, (k + 1) * ny),
                          source=(h * (k % nx), h * (k * ny + k % ny), 0.0), T=0) for k in which], h, out.data_ptr())
        return out.cpu().numpy().reshape(len(which), size)

    together = predict(range(n))
    assert np.isfinite(together).all() and (together > 0).any()
    for k in sorted({0, n // 2, n - 1}):
        np.testing.assert_array_equal(predict([k])[0], together[k])
    np.testing.assert_array_equal(predict(range(n - 2, n)), together[n - 2:])
    net.close()
