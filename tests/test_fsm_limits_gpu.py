"""The tiled sweeps of the Noble-Gesret-Belayouni operator against the plane schedule, bit for bit,
on models at the limits of their short arithmetic (both take the same updates in the same order,
the plane schedule with plain roots, divisions and std::min): nodes of zero or nearly zero
velocity scattered through the model, next to which a 2D candidate can have a negative
discriminant although its test holds (std::min then drops what follows it), and slownesses so
small that the root's argument leaves the short root's range.  One shot takes eight warps a tile;
many copies of it (more than 800 tiles on the widest diagonal) take one.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(tomo, slow, h, node, copies):
    ny, nx, nz = slow.shape
    with tomo.Context(nx, ny, nz, h) as ctx:
        ctx.set_slowness(slow)
        for shots in (1, copies):
            src = np.tile(np.float32(h) * np.array(node, np.float32), (shots, 1))
            ctx.eik_solve(src, op=1, sweep_groups=1)
            planes = ctx.eik_volume(0)
            ctx.eik_solve(src, op=1)
            for i in (0, shots - 1):
                np.testing.assert_array_equal(ctx.eik_volume(i), planes)


@pytest.mark.parametrize("velocity", [0.0, 1e-9], ids=str)
@pytest.mark.parametrize("seed", [12, 13, 20, 29, 33, 56])
def test_scattered_slow_nodes(tomo, velocity, seed):
    """On these models, which a serial restatement picked, a minimum that drops every NaN gives
    other times at 29 to 1,017 of the nodes."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = 24, 20, 16
    v = rng.uniform(1500.0, 2000.0, (ny, nx, nz)).astype(np.float32)
    v[rng.random(v.shape) < 0.5] = velocity
    node = (rng.integers(1, nx - 3), rng.integers(1, ny - 3), rng.integers(0, nz - 3))
    with np.errstate(divide="ignore"):
        _both(tomo, np.float32(1.0) / v, 25.0, node, 240)


@pytest.mark.parametrize("exponent", [-64, -60, -54, -36, -35, -34, 30], ids=str)
def test_tiny_slowness(tomo, exponent):
    """Root arguments of about 2^(2 exponent - 7); at this spacing the short forms take slownesses from
    2^-34.9 up."""
    slow = (np.random.default_rng(abs(exponent)).uniform(1.0, 2.0, (44, 60, 30)) * 2.0 ** exponent).astype(np.float32)
    _both(tomo, slow, 25.0, (7, 30, 0), 90)
