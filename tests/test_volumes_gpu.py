"""All fields of a solve in natural order (tomo_eik_volumes) against the fields one by one, on
depths and widths that end inside a block's 32 x 4 nodes, windows off the brick grid, and one
shot and many."""
import numpy as np
import pytest

from seismic_tomography_3d_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(5, 6, 2), (9, 8, 31), (12, 17, 32), (20, 21, 33), (33, 34, 70)], ids=str)
@pytest.mark.parametrize("shots,win", [(1, 0), (3, 1), (70, 0)], ids=["one", "windows", "many"])
def test_all_fields_at_once(tomo, n, shots, win):
    import torch

    nx, ny, nz = n
    sv = wl.small(sum(n), nx, ny, nz, nshots=shots, nrec=4)
    windows = None
    if win:
        sv.shots[:, :2] = np.maximum(sv.shots[:, :2], np.float32(sv.h))
        windows = np.array([[1, nx, 0, ny], [0, nx, 1, ny], [1, nx, 1, ny]], np.int32)
    with tomo.Context(nx, ny, nz, sv.h) as ctx:
        ctx.set_velocity(sv.velocity)
        ctx.eik_solve(sv.shots, windows=windows)
        sizes = ctx.volume_sizes(shots, windows)
        out = torch.full((sum(sizes) + 1,), -7.0, dtype=torch.float32, device="cuda")
        ctx.eik_volumes_to(out.data_ptr())
        got = out.cpu().numpy()
        assert got[-1] == -7.0
        at = 0
        for i, m in enumerate(sizes):
            np.testing.assert_array_equal(got[at:at + m], ctx.eik_volume(i).ravel())
            at += m
