"""Depth planes at a non-finite depth: 0 * depth makes that plane's points NaN (int(NaN) is
bin 0, like the reference's cast) and no other plane's, wherever it stands in a block of
16 planes; the last place, which also stands in for the planes beyond the end, included.
Against the kernel that reads the rows from global memory, to 1e-6 relative L2."""
import numpy as np
import pytest

from tests.conftest import rel_l2
from tests.test_depth_tiles_gpu import _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,flat", [(17, True), (17, False)])
@pytest.mark.parametrize("D,at", [(1, 0), (3, 2), (5, 0), (16, 15), (20, 15), (20, 19)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_a_non_finite_depth_stays_in_its_plane(ctx, cuda, side, flat, D, at, value):
    rng = np.random.default_rng(D + at)
    L, T = side * side, 256
    gx, gz = np.meshgrid(np.linspace(-1, 1, side), np.linspace(-1, 1, side))
    y = np.zeros(L) if flat else rng.uniform(-0.01, 0.01, L)
    xyz = np.stack([gx.ravel(), y, gz.ravel()], axis=1).astype(np.float32)
    depths = np.linspace(0.3, 1.2, D)
    depths[at] = value
    cube = rng.poisson(3.0, (L, T)).astype(np.float32)
    got, want = _pair(ctx, cuda, L, T, depths, (0, -1, 0), False, 0.0, 1, xyz, cube)
    assert want.any()
    for d in range(D):
        assert rel_l2(got[:, d], want[:, d]) < 1e-6, d


@pytest.mark.parametrize("normal", [(0, -1, 0), (0.36, -0.8, 0.48)])
def test_few_planes_of_many_points_go_by_rows(ctx, cuda, normal):
    """Tiles work on 16 planes whatever their number: two planes of 240^2 scan points take the row
    kernel, the bits of a capture with too many (zero) bins for tiles, sixteen the tiles."""
    import torch

    from fasterbackprojection_gb300 import make_info

    side, T, most = 240, 64, 3700
    L = side * side
    gx, gz = np.meshgrid(np.linspace(-1, 1, side), np.linspace(-1, 1, side))
    xyz = torch.from_numpy(np.stack([gx.ravel(), np.zeros(L), gz.ravel()], axis=1).astype(np.float32)).to(cuda)
    cube = torch.zeros((L, most), device=cuda)
    cube[:, :T] = torch.rand((L, T), generator=torch.Generator(device=cuda).manual_seed(1), device=cuda)
    depths = torch.linspace(0.3, 1.2, 16, dtype=torch.float64, device=cuda)

    def planes(bins, n):
        info = make_info(num_laser_targets=L, num_time_bins=bins, time_step=4.0 / T, voxel_res=(1, 1, 1),
                         hidden_min=(0, 0, 0), voxel_size=(1, 1, 1), wall_normal=normal)
        return ctx.backproject_depths(info, cube[:, :bins].contiguous(), xyz, depths[:n].contiguous())

    assert torch.equal(planes(T, 2), planes(most, 2))
    got, want = planes(T, 16), planes(most, 16)
    ctx.check_device_status()
    assert bool(want.any()) and not torch.equal(got, want)
    assert rel_l2(got.cpu().numpy(), want.cpu().numpy()) < 1e-6
