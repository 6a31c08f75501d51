"""Which kernel a batch is solved with (tomo_eik_kernel): one thread-block cluster per shot for up
to four shots that fit a cluster, the grid-wide kernels for everything else, two bricks per warp
from 2^20 bricks on -- also from several host threads at once, each with its own context and shots
of its own size.
"""
import threading

import numpy as np
import pytest

from seismic_tomography_3d_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _kernel(tomo, n, shots, windows=None, **kw):
    sv = wl.small(3, *n, nshots=shots)
    with tomo.Context(*n, sv.h) as ctx:
        assert ctx.eik_kernel() is None
        ctx.set_velocity(sv.velocity)
        ctx.eik_solve(sv.shots, **kw)
        return ctx.eik_kernel()


@pytest.mark.parametrize("n,shots,options,kernel", [
    ((4, 4, 4), 1, {}, "k_fim_cluster"),
    ((60, 60, 60), 4, {}, "k_fim_cluster"),
    ((60, 60, 60), 5, {}, "k_fim_solve"),         # five shots
    ((140, 128, 48), 1, {}, "k_fim_solve"),       # 13,440 bricks
    ((60, 60, 60), 1, dict(time_band=0.1), "k_fim_pair"),
    ((60, 60, 60), 1, dict(schedule=1), "k_fim_solve"),
    ((60, 60, 60), 1, dict(schedule=2), "k_fim_async"),
    ((60, 60, 60), 1, dict(block_warps=8), "k_fim_solve"),
    ((60, 60, 60), 1, dict(occupancy=3), "k_fim_solve"),
    ((60, 60, 60), 1, dict(spin_limit=1 << 20), "k_fim_solve"),
    ((60, 60, 60), 1, dict(brick=2), "k_fim_solve8"),
    ((60, 60, 60), 1, dict(op=1), "k_fsm"),
    ((256, 256, 64), 15, {}, "k_fim_solve"),      # 983,040 bricks
    ((256, 256, 64), 16, {}, "k_fim_pair"),       # 2^20 bricks
    ((256, 256, 64), 16, dict(schedule=1), "k_fim_solve"),
], ids=str)
def test_kernel_of_a_batch(tomo, n, shots, options, kernel):
    assert _kernel(tomo, n, shots, **options) == kernel


def test_contexts_on_threads_keep_their_clusters(tomo):
    sizes, errors = [(8, 8, 8)] * 7 + [(80, 80, 60)] * 3, []
    kernels = [set() for _ in sizes]

    def work(i):
        try:
            sv = wl.small(3 + i, *sizes[i])
            with tomo.Context(*sizes[i], sv.h) as ctx:
                ctx.set_velocity(sv.velocity)
                for _ in range(4000):
                    ctx.eik_solve(sv.shots)
                    kernels[i].add(ctx.eik_kernel())
        except Exception as e:  # reported below, on the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert kernels == [{"k_fim_cluster"}] * len(sizes)


def test_iteration_reports_its_solve(tomo):
    """Also when the solve is replayed from a graph after another kernel ran."""
    n = (40, 36, 24)
    sv = wl.small(2, *n, nshots=2, nrec=9)
    with tomo.Context(*n, sv.h) as ctx:
        ctx.set_velocity(sv.velocity)
        t, _ = ctx.eik_solve(sv.shots, receivers=sv.receivers, op=1)
        ctx.set_observed(t * np.float32(1.01))
        for _ in range(3):
            ctx.eik_solve(sv.shots, receivers=sv.receivers, op=1)
            assert ctx.eik_kernel() == "k_fsm"
            ctx.iteration(sv.shots, sv.receivers, (2 * sv.h,) * 3, cg_iterations=3)
            assert ctx.eik_kernel() == "k_fim_cluster"


def test_autotuned_context_keeps_clusters(tomo):
    """A shape tuned on a batch that clusters solve faster is not kept; one tuned on a larger
    batch leaves the small batches their clusters; what the caller asks for is always taken."""
    small, n = wl.small(3, 33, 29, 17), (33, 29, 17)
    with tomo.Context(*n, small.h) as ctx:
        ctx.set_velocity(small.velocity)
        _, st = ctx.eik_autotune(small.shots)
        assert 0 < st["best_ms"] <= st["default_ms"]
        ctx.eik_solve(small.shots)
        assert ctx.eik_kernel() == "k_fim_cluster"
    many = wl.small(3, 60, 60, 40, nshots=24)
    with tomo.Context(60, 60, 40, many.h) as ctx:
        ctx.set_velocity(many.velocity)
        shape, st = ctx.eik_autotune(many.shots)
        assert 0 < st["best_ms"] <= st["default_ms"]
        banded = st["best_ms"] < st["default_ms"] and shape["time_band"] > 0
        ctx.eik_solve(many.shots[:2])
        # a tuned time band applies to every later solve, and clusters run without one
        assert ctx.eik_kernel() == ("k_fim_pair" if banded else "k_fim_cluster")
        T = ctx.eik_volume(1)
        ctx.eik_solve(many.shots[:2], schedule=1, brick=1)
        assert ctx.eik_kernel() == "k_fim_solve"
        np.testing.assert_allclose(ctx.eik_volume(1), T, rtol=1e-5, atol=1e-6)
        ctx.eik_solve(many.shots)
        assert ctx.eik_kernel() != "k_fim_cluster"
