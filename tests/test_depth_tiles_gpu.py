"""The tiled confocal depth planes against the kernel that reads the rows from
global memory, one thread per test point: the same capture with zero bins
appended (rows too long for windows) takes that kernel.  Bins are the same
FP32 expression in both, so only the order of the FP32 sums differs: 1e-6
relative L2 (blocks of 32 and 64 terms, compensated across blocks)."""
import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

# scan points, bins, depths, wall normal, bounces kept, time offset, layout:
# grids of one tile, of a ragged second one and of none (37, 300 points);
# depth blocks of 1, 16 and 17; windows narrower than the row and the row.
CASES = [
    (1, 8, 1, (0, -1, 0), False, 0.0, 1),
    (37, 512, 16, (0, -1, 0), False, 0.0, 1),
    (256, 1024, 17, (0, -1, 0), True, 0.0, 0),
    (324, 700, 33, (0, -1, 0), False, 0.6, 1),
    (300, 96, 40, (0.36, -0.8, 0.48), True, 0.3, 1),
    (625, 2048, 20, (0.6, -0.8, 0.0), False, -0.2, 0),
]


def _pair(ctx, cuda, L, T, depths, normal, bounce, t0, layout, xyz, cube):
    import torch

    from fasterbackprojection_gb300 import make_info

    out = []
    for bins in (T, 6000):
        c = np.zeros((L, bins), np.float32)
        c[:, :T] = cube
        info = make_info(num_laser_targets=L, num_time_bins=bins, time_step=4.0 / T, voxel_res=(1, 1, 1),
                         hidden_min=(0, 0, 0), voxel_size=(1, 1, 1), wall_normal=normal, time_offset=t0,
                         discard_first_last_bounces=0 if bounce else 1, laser_position=(0.05, -0.25, 0.1),
                         sensor_position=(-0.1, -0.2, 0.05))
        d = torch.from_numpy(c if layout == 1 else np.ascontiguousarray(c.T)).to(cuda)
        got = ctx.backproject_depths(info, d, torch.from_numpy(xyz).to(cuda), torch.from_numpy(depths).to(cuda),
                                     layout=layout)
        out.append(got.cpu().numpy())
    ctx.check_device_status()
    return out


@pytest.mark.parametrize("L,T,D,normal,bounce,t0,layout", CASES)
def test_tiles_equal_the_row_kernel(ctx, cuda, L, T, D, normal, bounce, t0, layout):
    rng = np.random.default_rng(L + T)
    side = int(round(L ** 0.5))
    if side * side == L:
        gx, gz = np.meshgrid(np.linspace(-1, 1, side), np.linspace(-1, 1, side))
        xyz = np.stack([gx.ravel(), rng.uniform(-0.01, 0.01, L), gz.ravel()], axis=1).astype(np.float32)
    else:
        xyz = rng.uniform(-1, 1, (L, 3)).astype(np.float32) * np.float32([1, 0.01, 1])
    cube = rng.poisson(3.0, (L, T)).astype(np.float32)
    cube[rng.random((L, T)) < 0.3] = 5e-6  # at or below the threshold: skipped
    got, want = _pair(ctx, cuda, L, T, rng.uniform(0.0, 1.2, D), normal, bounce, t0, layout, xyz, cube)
    assert want.any()
    assert rel_l2(got, want) < 1e-6


def test_non_finite_points_and_depths(ctx, cuda):
    """int(NaN) is bin 0, int(inf) is past the last bin, in both kernels."""
    rng = np.random.default_rng(5)
    L, T = 289, 256
    gx, gz = np.meshgrid(np.linspace(-1, 1, 17), np.linspace(-1, 1, 17))
    xyz = np.stack([gx.ravel(), np.zeros(L), gz.ravel()], axis=1).astype(np.float32)
    xyz[40, 1] = np.nan
    xyz[200, 0] = np.inf
    depths = np.array([0.3, np.inf, 0.7, np.nan, 0.9])
    cube = rng.poisson(3.0, (L, T)).astype(np.float32)
    got, want = _pair(ctx, cuda, L, T, depths, (0, -1, 0), False, 0.0, 1, xyz, cube)
    assert rel_l2(got, want) < 1e-6
