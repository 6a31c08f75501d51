"""The surrogate's kernels at the limits of what they accept.

Predicted traveltimes far outside metres: everything that the prediction forms scales by a power
of two with the spacing, so the times at a spacing of 2^e h are those at h times 2^e, bit for bit,
also where squared distances leave the short root's range.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [-64, -52, 40, 58], ids=str)
@pytest.mark.parametrize("stride", [1, 3])
def test_times_scale_with_the_spacing(tomo, exponent, stride):
    import torch

    nx, ny, nz = 21, 18, 15
    slow = torch.from_numpy(np.random.default_rng(3).uniform(2e-4, 6e-4, (ny, nx, nz)).astype(np.float32)).cuda()
    out = torch.zeros(2, nx * ny * nz, dtype=torch.float32, device="cuda")
    net = tomo.Net(seed=2)
    for i, h in enumerate((1.0, 2.0 ** exponent)):
        net.predict([dict(slow=slow.data_ptr(), model_nx=nx, model_ny=ny, nz=nz, window=(0, nx, 0, ny), T=0,
                          source=(4 * h, 3 * h, 0.0))], h, out[i].data_ptr(), stride=stride)
    net.close()
    assert (out[0] != 0).float().mean() > 0.9
    np.testing.assert_array_equal(out[1].cpu().numpy(), out[0].cpu().numpy() * np.float32(2.0 ** exponent))
