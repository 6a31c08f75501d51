"""Small batches solve with one thread-block cluster per shot (at most 4 shots of at most about
12,000 bricks, nothing of the launch asked for); more shots, larger ones or an explicit schedule
take the grid-wide kernel.  Both reach the same fixed point: with every drop re-queued
(change_tol < 0) the fields agree to FP32 rounding of the last updates (1e-6), on brick counts
that are and are not multiples of the cluster's 16 CTAs, windows on and off the brick grid, and
sizes on both sides of the limits.
"""
import numpy as np
import pytest

from seismic_tomography_3d_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _fields(ctx, shots, n, **kw):
    t, st = ctx.eik_solve(shots, change_tol=-1.0, **kw)
    return t, st, [ctx.eik_volume(i) for i in range(n)]


@pytest.mark.parametrize("n,shots", [((4, 4, 4), 1), ((5, 9, 2), 2), ((16, 16, 16), 4), ((33, 29, 17), 1), ((33, 29, 17), 5),
                                     ((60, 60, 60), 2), ((101, 97, 51), 1), ((120, 128, 48), 1), ((140, 128, 48), 1)], ids=str)
@pytest.mark.parametrize("windows", [None, "aligned", "any"])
def test_same_fixed_point(tomo, n, shots, windows):
    nx, ny, nz = n
    if windows and min(nx, ny) < 16:
        pytest.skip("no window inside")
    sv = wl.small(nx + shots, nx, ny, nz, nshots=shots, nrec=min(20, nx * ny // 2))
    win = None
    if windows:
        a = 4 if windows == "aligned" else 3
        win = np.array([[a, nx, a, ny]] * shots, np.int32)
        sv.shots[:, :2] = np.maximum(sv.shots[:, :2], np.float32((a + 1) * sv.h))
    with tomo.Context(nx, ny, nz, sv.h) as ctx:
        ctx.set_velocity(sv.velocity)
        t, st, here = _fields(ctx, sv.shots, shots, windows=win, receivers=sv.receivers)
        t1, st1, rounds = _fields(ctx, sv.shots, shots, windows=win, receivers=sv.receivers, schedule=1)
    assert st["rounds"] > 0 and st["activations"] > 0 and st["nodes_per_brick"] == st1["nodes_per_brick"]
    for a, b in zip(here, rounds):
        np.testing.assert_allclose(a, b, rtol=1e-6, atol=1e-7)
    np.testing.assert_allclose(t, t1, rtol=2e-6, atol=1e-7)


def test_round_cap_and_recovery(tomo):
    sv = wl.small(4, 33, 29, 17, nshots=2, nrec=8)
    with tomo.Context(33, 29, 17, sv.h) as ctx:
        ctx.set_velocity(sv.velocity)
        with pytest.raises(tomo.TomoError) as e:
            ctx.eik_solve(sv.shots, max_rounds=2)
        assert e.value.status == -4
        _, _, a = _fields(ctx, sv.shots, 2)
        _, _, b = _fields(ctx, sv.shots, 2, schedule=1)
        for x, y in zip(a, b):
            np.testing.assert_allclose(x, y, rtol=1e-6, atol=1e-7)
