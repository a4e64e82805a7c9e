"""Exhaustive captures whose windows leave room for two of them in a CTA's shared memory, not
three (some 17,700 bins and more), on both sides of that line, against the FP64 oracle with the
GPU's bins: 1e-6 relative L2, the bound of the gather's sums of 32 terms and compensated folds.
Windows that are the whole row and, with more bins than a tile's paths can reach, that are not."""
import numpy as np
import pytest

from oracle import cpu
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _run(ctx, cuda, T, vres, size, bounce, t0, dt):
    import torch

    from fasterbackprojection_gb300 import FBP_EXHAUSTIVE, make_info, scenes

    nl, ns = 2, 3
    cap = scenes.exhaustive_points(nl, ns, T, dt / scenes.LIGHT_SPEED, n_points=60, depth_range=(0.3, 1.3), seed=T)
    rng = np.random.default_rng(T)
    cube = (cap.cube + rng.poisson(0.5, cap.cube.shape)).astype(np.float32)
    info = make_info(num_laser_targets=nl * nl, num_sensor_targets=ns * ns, num_time_bins=T, time_step=dt,
                     voxel_res=vres, hidden_min=(-size[0] / 2, -0.1 - size[1], -size[2] / 2),
                     voxel_size=(size[0] / vres[0], size[1] / vres[2], size[2] / vres[1]), capture_system=FBP_EXHAUSTIVE,
                     discard_first_last_bounces=0 if bounce else 1, time_offset=t0,
                     laser_position=(0.05, -0.25, 0.1), sensor_position=(-0.1, -0.2, 0.05))
    lx, sx = torch.from_numpy(cap.laser_xyz).to(cuda), torch.from_numpy(cap.sensor_xyz).to(cuda)
    vol = ctx.backproject_exhaustive(info, torch.from_numpy(cube).to(cuda), lx, sx)
    bins = ctx.debug_exhaustive_bins(info, lx, sx, torch.arange(vol.numel(), device=cuda)).cpu().numpy()
    ctx.check_device_status()
    want = cpu.exhaustive_voxel(info, cube, cap.laser_xyz, cap.sensor_xyz, bins=bins)
    assert (bins >= 0).any()
    assert rel_l2(vol.cpu().numpy(), want) < 1e-6


@pytest.mark.parametrize("bounce,t0", [(False, 0.0), (True, 0.0), (False, 0.4), (False, -0.2)])
@pytest.mark.parametrize("T", [17720, 17728, 18636, 26500])
def test_whole_rows(ctx, cuda, T, bounce, t0):
    _run(ctx, cuda, T, (9, 5, 6), (2.0, 1.4, 2.0), bounce, t0, 4.92 / T)


@pytest.mark.parametrize("bounce,t0", [(False, 0.0), (True, 0.4)])
@pytest.mark.parametrize("span", [17000, 18200])
def test_part_of_the_row(ctx, cuda, span, bounce, t0):
    size = (0.5, 0.4, 0.4)  # one tile; its diagonal, there and back, spans `span` bins
    _run(ctx, cuda, 60000, (8, 4, 4), size, bounce, t0, 2 * float(np.linalg.norm(size)) / span)


def test_wider_windows_are_refused(ctx, cuda):
    from fasterbackprojection_gb300._lib import FbpError

    with pytest.raises(FbpError, match="too large"):
        _run(ctx, cuda, 27000, (9, 5, 6), (2.0, 1.4, 2.0), False, 0.0, 4.92 / 27000)
