"""The tiled sweeps of the Noble-Gesret-Belayouni operator, bit for bit against the oracle, on
both sides of what they choose by: one warp per tile (many tiles on a diagonal) and eight (few),
sizes at the edges of the 16 x 8 x 8 tiles, unequal spacings, spacings the short division does
not take, and zero velocity (infinite slowness).  NaN in the model takes the plain arithmetic
in std::min's order, which the oracle does not restate: there the tiles must give what the
plane schedule gives.
"""
import numpy as np
import pytest

from seismic_tomography_3d_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _check(tomo, oracle_mod, slow, h, shots, which):
    ny, nx, nz = slow.shape
    with tomo.Context(nx, ny, nz, *(h if np.ndim(h) else (h,))) as ctx:
        ctx.set_slowness(slow)
        ctx.eik_solve(shots, op=1)
        got = [ctx.eik_volume(i) for i in which]
    for i, T in zip(which, got):
        ref = oracle_mod.fsm_ngb(slow, h, tuple(map(float, shots[i])))
        np.testing.assert_array_equal(T, ref[0] if isinstance(ref, tuple) else ref)


@pytest.mark.parametrize("n", [(6, 6, 14), (7, 8, 15), (9, 15, 16), (23, 24, 31), (40, 17, 46)], ids=str)
@pytest.mark.parametrize("shots", [1, 3])
def test_edges_of_tiles(tomo, oracle_mod, n, shots):
    sv = wl.small(n[0], *n, nshots=shots)
    src = np.minimum(sv.shots, np.float32(sv.h) * (np.array(n, np.float32) - 3))  # off the far faces
    _check(tomo, oracle_mod, (1.0 / sv.velocity).astype(np.float32), sv.h, src.astype(np.float32), range(shots))


def test_many_tiles_on_a_diagonal(tomo, oracle_mod):
    """64 shots: one warp per tile (more than 800 tiles on the widest diagonal)."""
    sv = wl.small(5, 60, 55, 30, nshots=64)
    src = np.minimum(sv.shots, np.float32(sv.h) * np.array([57, 52, 27], np.float32)).astype(np.float32)
    _check(tomo, oracle_mod, (1.0 / sv.velocity).astype(np.float32), sv.h, src, [0, 17, 63])


@pytest.mark.parametrize("h", [(25.0, 20.0, 10.0), 2.0 ** 21, 2.0 ** -21], ids=str)
def test_spacings(tomo, oracle_mod, h):
    sv = wl.small(7, 21, 18, 17, nshots=2)
    d = np.array(h if np.ndim(h) else (h,) * 3, np.float32)
    src = (np.array([[4, 5, 0], [11, 9, 3]], np.float32) * d).astype(np.float32)
    _check(tomo, oracle_mod, (1.0 / sv.velocity).astype(np.float32), tuple(map(float, d)), src, range(2))


def _special(value, shots):
    sv = wl.small(8, 60, 44, 30, nshots=shots)
    slow = (1.0 / sv.velocity).astype(np.float32)
    slow[10:16, 20:31, 5:12] = value
    slow[30, 40, 20] = value
    return slow, sv.h, np.minimum(sv.shots, np.float32(sv.h) * np.array([57, 41, 27], np.float32)).astype(np.float32)


@pytest.mark.parametrize("value", [np.inf, 0.0], ids=str)
@pytest.mark.parametrize("shots", [1, 40])
def test_special_slowness(tomo, oracle_mod, value, shots):
    slow, h, src = _special(value, shots)
    _check(tomo, oracle_mod, slow, h, src, [0, shots - 1])


@pytest.mark.parametrize("shots", [1, 40])
def test_nan_slowness(tomo, shots):
    slow, h, src = _special(np.nan, shots)
    with tomo.Context(60, 44, 30, h) as ctx:
        ctx.set_slowness(slow)
        ctx.eik_solve(src, op=1)
        tiles = [ctx.eik_volume(i) for i in (0, shots - 1)]
        ctx.eik_solve(src, op=1, sweep_groups=1)
        for i, T in zip((0, shots - 1), tiles):
            np.testing.assert_array_equal(T, ctx.eik_volume(i))
