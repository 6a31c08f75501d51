"""The surrogate's kernels at the limits of what they accept.

Predicted traveltimes far outside metres: everything that the prediction forms scales by a power
of two with the spacing, so the times at a spacing of 2^e h are those at h times 2^e, bit for bit,
also where squared distances leave the short root's range.

A sample without a single target (all its traveltimes 0) takes no part in the loss: the head's
gradient is the other sample's alone, also where the untargeted sample's activations overflow.

A window whose vertical section has more than 2^31 nodes is predicted in full.
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


def _offsets(spec):
    at, out = 0, []
    for cin, cout in spec:
        out.append((at, cin))
        at += 27 * cin * cout + cout
    return out, at


def test_untargeted_sample_leaves_the_head_alone(tomo):
    import torch

    n, h = 8, 10.0
    spec = [(16, 16), (16, 16), (16, 32), (32, 32), (32, 48), (48, 48), (48, 64), (64, 64), (112, 48), (48, 48),
            (80, 32), (32, 32), (48, 16), (16, 16)]
    where, head = _offsets(spec)
    net = tomo.Net(seed=2)
    p = np.zeros(len(net.get_params()), np.float32)
    assert head + 17 == len(p)

    def centre(layer, ci, value):  # output channel 0 of a layer reads input channel ci alone
        off, cin = where[layer]
        p[off + 13 * cin + ci] = value

    # slowness contrast -> first level -> skip connection -> head, times 1e20 in the last layer
    centre(0, 0, 1.0)
    centre(1, 0, 1.0)
    centre(12, 32, 1.0)
    centre(13, 0, 1e20)
    p[head] = 1e-20
    net.set_params(p)
    slow = np.full((2, n, n, n), 4e-4, np.float32)
    slow[0, :, :, 4:] = 8e-4  # contrast 1: activations up to 1e20
    slow[1, :, :, 4:] = 4e26  # contrast 1e30: 1e50 in the last layer
    d = np.sqrt(sum(a.astype(np.float64) ** 2 for a in np.meshgrid(*[np.arange(n)] * 3, indexing="ij"))) * h
    times = np.zeros((2, n, n, n), np.float32)
    times[0] = 5e-4 * d
    sd, td = torch.from_numpy(slow).cuda(), torch.from_numpy(times).cuda()
    samples = [dict(slow=sd[i].data_ptr(), model_nx=n, model_ny=n, nz=n, window=(0, n, 0, n), source=(0.0, 0.0, 0.0),
                    T=td[i].data_ptr()) for i in range(2)]
    loss1, g1 = net.gradients(samples[:1], h)
    loss2, g2 = net.gradients(samples, h)
    net.close()
    assert 0 < loss1 < np.inf and loss1 == loss2
    assert np.isfinite(g1[head:]).all() and g1[head] != 0
    # the same sums in other groups: a few hundred terms, 6e-8 each
    np.testing.assert_allclose(g2[head:], g1[head:], rtol=1e-5, atol=0)


def test_more_than_2_31_nodes_in_a_section(tomo):
    import torch

    nx, ny, nz, h = 2, 46341, 46342, 10.0
    if torch.cuda.mem_get_info()[0] < 110e9:
        pytest.skip("needs 110 GB of device memory")
    slow = torch.full((ny, nx, nz), 4e-4, dtype=torch.float32, device="cuda")
    out = torch.full((ny, nx, nz), -7.0, dtype=torch.float32, device="cuda")
    net = tomo.Net(seed=2)
    net.predict([dict(slow=slow.data_ptr(), model_nx=nx, model_ny=ny, nz=nz, window=(0, nx, 0, ny), T=0,
                      source=(0.0, 0.0, 0.0))], h, out.data_ptr(), stride=16)
    net.close()
    missing = sum(int((out[k:k + 4096] == -7.0).sum()) for k in range(0, ny, 4096))
    corner = [float(out[y, 0, z]) / (4e-4 * h * (y * y + z * z) ** 0.5) for y, z in ((ny - 1, nz - 1), (ny - 1, 0), (0, nz - 1))]
    del slow, out
    torch.cuda.empty_cache()
    assert missing == 0
    assert np.isfinite(corner).all() and 0.0 not in corner
