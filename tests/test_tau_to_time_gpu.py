"""Predicted traveltimes at the nodes between the network's samples: T / (s_src distance)
must be the trilinear interpolation of its values at the sampled nodes, for windows that end
inside a cell, on one, or within a run of nodes along x, and for several windows in one call.

Tolerance: about 20 FP32 roundings (6e-8 each) lie between the two sides.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 4e-6


def _axis(n, k):
    """(lower sample, upper sample, weight) of every node of an axis."""
    x, nc = np.arange(n), -(-n // k)
    c0 = np.minimum(x // k, nc - 1)
    c1 = np.minimum(c0 + 1, nc - 1)
    p0, p1 = c0 * k, np.minimum(c1 * k, n - 1)
    return c0, c1, np.where(p1 > p0, (x - p0) / np.maximum(p1 - p0, 1), 0.0)


@pytest.mark.parametrize("shape", [(33, 7, 5, 2), (32, 9, 17, 4), (65, 18, 3, 16), (70, 13, 31, 3), (40, 6, 9, 8),
                                   (97, 33, 34, 5), (8, 40, 11, 4)], ids=str)
def test_times_between_samples_are_interpolated(tomo, shape):
    import torch

    nx, ny, nz, k = shape
    h, windows = 10.0, [(0, nx, 0, ny), (0, nx - 1, 0, ny - 1)]
    rng = np.random.default_rng(nx)
    slow = rng.uniform(2e-4, 6e-4, (ny, nx, nz)).astype(np.float32)
    sd = torch.from_numpy(slow).cuda()
    src = (h, h, 0.0)  # off every sample: two of its indices are no multiple of k
    sizes = [nz * (w[1] - w[0]) * (w[3] - w[2]) for w in windows]
    out = torch.full((sum(sizes) + 1,), -7.0, dtype=torch.float32, device="cuda")
    net = tomo.Net(seed=2)
    net.predict([dict(slow=sd.data_ptr(), model_nx=nx, model_ny=ny, nz=nz, window=w, source=src, T=0) for w in windows],
                h, out.data_ptr(), stride=k)
    net.close()
    got = out.cpu().numpy()
    assert got[-1] == -7.0
    s_src, at = float(slow[1, 1, 0]), 0
    for (x0, x1, y0, y1), n in zip(windows, sizes):
        T = got[at:at + n].reshape(y1 - y0, x1 - x0, nz).astype(np.float64)
        at += n
        g = np.meshgrid(*(np.arange(m) * h for m in T.shape), indexing="ij")
        dist = np.sqrt((g[0] - src[1]) ** 2 + (g[1] - src[0]) ** 2 + (g[2] - src[2]) ** 2)
        tau = (T / (s_src * np.maximum(dist, 1e-9)))[::k, ::k, ::k]
        for axis, m in enumerate(T.shape):
            c0, c1, w = _axis(m, k)
            w = w.reshape([-1 if a == axis else 1 for a in range(3)])
            tau = tau.take(c0, axis) * (1 - w) + tau.take(c1, axis) * w
        far = dist >= h * (1 + 1e-6)
        near = dist < h * (1 - 1e-6)
        np.testing.assert_allclose(T[far], (tau * s_src * dist)[far], rtol=RTOL, atol=0)
        assert not T[near].any()
