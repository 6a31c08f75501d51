"""The model update on sizes at the edges of its tiles (32 x 16 x 8 nodes) and with every
filter it sums by itself or not, bit for bit against the oracle; and with the masks off,
where the far faces move and the padding of the brick-major model has to follow them: a
solve afterwards equals one on a fresh context that is given the same slowness.
"""
import numpy as np
import pytest

from seismic_tomography_3d_b200 import workloads as wl

pytestmark = pytest.mark.gpu

H, D = 25.0, (60.0, 60.0, 60.0)


def _solution(tomo, nx, ny, nz):
    """A context with a CGLS solution, its starting slowness and the solution."""
    sv = wl.small(3, nx, ny, nz, h=H, nshots=2, nrec=24)
    ctx = tomo.Context(nx, ny, nz, H)
    ctx.set_velocity(sv.velocity)
    t, _ = ctx.eik_solve(sv.shots, receivers=sv.receivers)
    ctx.set_observed(t * np.float32(1.05))
    ctx.build_jacobian(D, max_ray_steps=4000)
    x, _, _ = ctx.cgls(4)
    return ctx, sv, (np.float32(1.0) / sv.velocity).astype(np.float32), x


def _cells(nx, ny, nz):
    return [int(np.float32((n - 1) * np.float32(H)) / np.float32(d)) + 1 for n, d in zip((nx, ny, nz), D)]


@pytest.mark.parametrize("samples", [0, 1, 3, 5, 7, 9])
@pytest.mark.parametrize("shape", [(49, 41, 33), (50, 47, 64), (34, 33, 20)], ids=str)
def test_update_is_the_oracles(tomo, oracle_mod, shape, samples):
    ctx, _, s0, x = _solution(tomo, *shape)
    with ctx:
        vel = ctx.model_update(smooth=samples > 0, filter_samples=max(samples, 1), standard_deviation=1.5)
        s = ctx.get_slowness()
    s_o, vel_o = oracle_mod.model_update(s0, H, D, _cells(*shape), x, samples > 0, max(samples, 1), 1.5)
    np.testing.assert_array_equal(s, s_o)
    np.testing.assert_array_equal(vel, vel_o)


@pytest.mark.parametrize("shape", [(33, 29, 17), (20, 18, 34), (35, 34, 31)], ids=str)
@pytest.mark.parametrize("smooth", [True, False])
def test_bricks_follow_the_model(tomo, shape, smooth):
    ctx, sv, _, _ = _solution(tomo, *shape)
    with ctx:
        ctx.model_update(smooth=smooth, reference_masks=False, want_velocity=False)
        s = ctx.get_slowness()
        ctx.eik_solve(sv.shots)
        T = [ctx.eik_volume(i) for i in range(len(sv.shots))]
    with tomo.Context(*shape, H) as fresh:
        fresh.set_slowness(s)
        fresh.eik_solve(sv.shots)
        for i, t in enumerate(T):  # the face tolerance lets the schedule move the last bits
            np.testing.assert_allclose(t, fresh.eik_volume(i), rtol=1e-5, atol=2e-6)
