"""An infinite sample of the last scan points (or pairs) makes the voxels that read it
infinite, not NaN, also where the points are walked in several chains whose sums are folded
afterwards; every other voxel keeps the bits it has without that sample."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _three(call, cube, at):
    """Volumes with the sample `at` zero, large and infinite."""
    out = []
    for value in (0.0, 6e4, float("inf")):
        c = cube.clone()
        c.view(-1)[at] = value
        out.append(call(c))
    return out


def _check(zero, large, inf):
    import torch

    touched = large != zero
    assert bool(touched.any()) and not bool(touched.all())
    assert bool(torch.isinf(inf[touched]).all()) and bool((inf[touched] > 0).all())
    assert torch.equal(inf[~touched], zero[~touched])


@pytest.mark.parametrize("dtype", ["float16", "float32"])
@pytest.mark.parametrize("n,vres", [(20, (16, 64, 24)), (8, (17, 17, 17))])
def test_confocal_and_batch(ctx, cuda, n, vres, dtype):
    import torch

    from fasterbackprojection_gb300 import Batch, make_info, scenes

    L, T = n * n, 300
    hmin, vs = scenes.volume_geometry(vres, depth_range=(0.0, 1.6))
    info = make_info(num_laser_targets=L, num_time_bins=T, time_step=4.92 / T, voxel_res=vres, hidden_min=hmin,
                     voxel_size=vs)
    cube = torch.ones((L, T), device=cuda).to(getattr(torch, dtype))
    lx = torch.from_numpy(scenes.confocal_points(n, T, 32e-12, n_points=1, seed=0).laser_xyz).to(cuda)
    before = ctx.launches
    ctx.backproject_confocal(info, cube, lx)
    assert ctx.launches - before == 3  # rows, chains, fold

    def batched(c):
        vol = torch.empty(vres[::-1], device=cuda)
        b = Batch(ctx, [(info, c, lx, vol, 1)])
        b.run()
        torch.cuda.synchronize()
        b.close()
        return vol

    at = (L - 1) * T + 120
    for call in (lambda c: ctx.backproject_confocal(info, c, lx), batched):
        _check(*_three(call, cube, at))
    ctx.check_device_status()


def test_exhaustive(ctx, cuda):
    import torch

    from fasterbackprojection_gb300 import FBP_EXHAUSTIVE, make_info, scenes

    nl, ns, T, vres = 4, 6, 300, (16, 20, 24)
    cap = scenes.exhaustive_points(nl, ns, T, 32e-12, n_points=1, seed=0)
    hmin, vs = scenes.volume_geometry(vres, depth_range=(0.0, 1.6))
    info = make_info(num_laser_targets=nl * nl, num_sensor_targets=ns * ns, num_time_bins=T, time_step=4.92 / T,
                     voxel_res=vres, hidden_min=hmin, voxel_size=vs, capture_system=FBP_EXHAUSTIVE)
    lx, sx = torch.from_numpy(cap.laser_xyz).to(cuda), torch.from_numpy(cap.sensor_xyz).to(cuda)
    cube = torch.ones((nl * nl, ns * ns, T), device=cuda)
    at = (nl * nl * ns * ns - 1) * T + 120
    _check(*_three(lambda c: ctx.backproject_exhaustive(info, c, lx, sx), cube, at))


def test_depth_planes(ctx, cuda):
    import torch

    from fasterbackprojection_gb300 import make_info, scenes

    n, T = 20, 300
    L = n * n
    info = make_info(num_laser_targets=L, num_time_bins=T, time_step=4.92 / T, voxel_res=(1, 1, 1), hidden_min=(0, 0, 0),
                     voxel_size=(1, 1, 1))
    cube = torch.ones((L, T), device=cuda)
    lx = torch.from_numpy(scenes.confocal_points(n, T, 32e-12, n_points=1, seed=0).laser_xyz).to(cuda)
    depths = torch.linspace(0.3, 1.2, 20, dtype=torch.float64, device=cuda)
    _check(*_three(lambda c: ctx.backproject_depths(info, c, lx, depths), cube, (L - 1) * T + 120))
