"""The training gradient on sizes at the edges of its kernels' tiles: a batch of copies of one
sample has that sample's loss and gradient.  With 2 or 4 copies the loss gradient of every
voxel is halved or quartered exactly, through all BF16 roundings, so the two differ by the order
of the FP32 sums alone: at most 1e-5 of the whole gradient (sums of up to 4 x 10^5 terms of
either sign, 6e-8 each, in blocks).
"""
import numpy as np
import pytest

from seismic_tomography_3d_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [2, 4])
@pytest.mark.parametrize("shape", [(8, 8, 8), (9, 17, 5), (24, 16, 40), (65, 33, 31)], ids=str)
def test_copies_have_the_samples_gradient(tomo, shape, copies):
    import torch

    nx, ny, nz = shape
    sv = wl.small(5, nx, ny, nz, h=20.0, nshots=1)
    with tomo.Context(nx, ny, nz, 20.0) as ctx:
        ctx.set_velocity(sv.velocity)
        ctx.eik_solve(sv.shots)
        T = torch.from_numpy(ctx.eik_volume(0)).cuda()
    slow = torch.from_numpy((1.0 / sv.velocity).astype(np.float32)).cuda()
    sample = dict(slow=slow.data_ptr(), model_nx=nx, model_ny=ny, nz=nz, window=(0, nx, 0, ny), source=sv.shots[0],
                  T=T.data_ptr())
    net = tomo.Net(seed=6)
    loss1, g1 = net.gradients([sample], 20.0)
    loss, g = net.gradients([sample] * copies, 20.0)
    net.close()
    assert loss1 > 0 and abs(loss - loss1) <= 1e-9 * loss1
    assert np.linalg.norm(g.astype(np.float64) - g1) <= 1e-5 * np.linalg.norm(g1.astype(np.float64))
