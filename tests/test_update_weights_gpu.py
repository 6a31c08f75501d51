"""The model update with one-sample filters whose weight is 1, and whose weight is NaN because the
square of the standard deviation leaves the FP32 range, bit for bit against the oracle."""
import numpy as np
import pytest

from seismic_tomography_3d_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("samples,stdv", [(1, 2.0), (1, 0.0), (1, 1e-25), (1, 1e25), (3, 1e-25)], ids=str)
def test_weights_at_the_limits(tomo, oracle_mod, samples, stdv):
    n, h, d = (34, 33, 20), 25.0, (60.0, 60.0, 60.0)
    sv = wl.small(3, *n, h=h, nshots=2, nrec=24)
    with tomo.Context(*n, h) as ctx:
        ctx.set_velocity(sv.velocity)
        t, _ = ctx.eik_solve(sv.shots, receivers=sv.receivers)
        ctx.set_observed(t * np.float32(1.05))
        ctx.build_jacobian(d, max_ray_steps=4000)
        x, _, _ = ctx.cgls(4)
        ctx.model_update(smooth=True, filter_samples=samples, standard_deviation=stdv)
        s = ctx.get_slowness()
    cells = [int(np.float32((m - 1) * np.float32(h)) / np.float32(c)) + 1 for m, c in zip(n, d)]
    s_o, _ = oracle_mod.model_update((np.float32(1.0) / sv.velocity).astype(np.float32), h, d, cells, x, True, samples, stdv)
    np.testing.assert_array_equal(s, s_o)
