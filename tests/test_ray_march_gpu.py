"""The ray march against the oracle's ray tracer on the same fields, bit for bit, where its
branches part: fields of a single brick along an axis, rays that cross more than the four
cells kept in registers and come back to them (cells of about a node), a per-ray capacity
that some rays exceed, spacings outside the range of the prepared divisors, and unequal ones.
"""
import numpy as np
import pytest

from seismic_tomography_3d_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    dict(n=(21, 18, 9), h=25.0, d=(60.0, 60.0, 60.0)),
    dict(n=(40, 33, 17), h=10.0, d=(10.1, 9.7, 11.3)),
    dict(n=(40, 33, 17), h=10.0, d=(4.0, 4.0, 4.0), cap=24),
    dict(n=(33, 7, 4), h=2.0 ** -44, d=(2.0 ** -42, 2.0 ** -42, 2.0 ** -42)),
    dict(n=(24, 24, 12), h=2.0 ** 41, d=(2.0 ** 42, 2.0 ** 42, 2.0 ** 43)),
], ids=["coarse", "node_cells", "overflow", "tiny_spacing", "huge_spacing"])
def test_rows_are_the_oracles(tomo, oracle_mod, case):
    nx, ny, nz = case["n"]
    h, d = float(case["h"]), tuple(map(float, case["d"]))
    sv = wl.small(9, nx, ny, nz, h=25.0, nshots=2, nrec=40)
    shots, rec = (sv.shots * np.float32(h / 25.0)), (sv.receivers * np.float32(h / 25.0))
    steps, cap = 3000, case.get("cap", 0)
    nt = [int(np.float32((n - 1) * np.float32(h)) / np.float32(q)) + 1 for n, q in zip((nx, ny, nz), d)]
    with tomo.Context(nx, ny, nz, h) as ctx:
        ctx.set_velocity(sv.velocity)
        ctx.eik_solve(shots, receivers=rec)
        vols = [ctx.eik_volume(i) for i in range(2)]
        ctx.build_jacobian(d, tk_order=1, max_ray_steps=steps, max_cells_per_ray=cap)
        rp, cols, vals = ctx.jacobian()
        status = ctx.ray_status().reshape(2, -1)
    over = 0
    for i, sh in enumerate(shots):
        rt = oracle_mod.raytrace(vols[i], h, sh, *rec.T, d, nt, max_steps=steps)
        for r in range(len(rec)):
            a, b = rt["row_ptr"][r], rt["row_ptr"][r + 1]
            g0, g1 = rp[i * len(rec) + r], rp[i * len(rec) + r + 1]
            if status[i, r] == 5:  # more runs than the capacity: an empty row
                over += 1
                assert g0 == g1 and cap
                continue
            assert status[i, r] == rt["status"][r]
            np.testing.assert_array_equal(cols[g0:g1], rt["cols"][a:b])
            np.testing.assert_array_equal(vals[g0:g1], rt["vals"][a:b])
    assert (over > 0) == bool(cap)
