"""The voxel-scattering gather's forms: 8 voxels per thread in one chain or several, 16 where every
walk is as long as its unrolled steps and the volume needs no chains; walks of 2, 3, 4 and more
steps, predicated or not, windows that are the whole row and that are not; volumes of fewer than 8
columns, of 8 and of one more.

Against the FP64 sum over the same walks (the GPU's paths), voxel by voxel (a sample of them where
there are many): FP32 sums of 32 scan points' steps, one rounding for each product and sum, folded
with compensation: (32 steps + 4) 2^-24 of the voxel's value, all terms being positive.  Voxels with a path
so short that its weight is the largest float are left out: their sums overflow."""
import numpy as np
import pytest

from oracle import numpy_ref

pytestmark = pytest.mark.gpu

# scan side, bins, volume, bounces kept, time offset
CASES = [
    (6, 200, (1, 9, 17), False, 0.0), (6, 200, (8, 16, 16), True, 0.3), (9, 500, (9, 17, 16), False, -0.2),
    (12, 128, (40, 40, 40), False, 0.0), (12, 300, (48, 40, 33), True, 0.0), (5, 2048, (24, 24, 24), False, 0.4),
    # no chains: one group of scan points, or tiles enough
    (5, 400, (96, 96, 96), False, 0.0), (5, 300, (96, 96, 96), True, 0.0), (4, 512, (112, 112, 96), False, -0.1),
    (5, 1200, (96, 96, 96), False, 0.0), (3, 200, (128, 64, 64), False, 0.2),
]


@pytest.mark.parametrize("n,T,vres,bounce,t0", CASES)
def test_scatter_forms(ctx, cuda, n, T, vres, bounce, t0):
    import torch

    from fasterbackprojection_gb300 import make_info, scenes

    cap = scenes.confocal_points(n, T, 4.92 / T / scenes.LIGHT_SPEED, n_points=60, depth_range=(0.3, 1.3), seed=n + T)
    cube = (cap.cube + np.random.default_rng(T).poisson(0.5, cap.cube.shape)).astype(np.float32)
    hmin, vs = scenes.volume_geometry(vres, depth_range=(0.0, 1.6))
    info = make_info(num_laser_targets=n * n, num_time_bins=T, time_step=cap.time_step, voxel_res=vres,
                     hidden_min=hmin, voxel_size=vs, discard_first_last_bounces=0 if bounce else 1, time_offset=t0,
                     laser_position=(0.05, -0.25, 0.1), sensor_position=(-0.1, -0.2, 0.05))
    lx = torch.from_numpy(cap.laser_xyz).to(cuda)
    got = ctx.backproject_confocal_scatter(info, torch.from_numpy(cube).to(cuda), lx).view(-1)
    V = got.numel()
    pick = torch.arange(V) if V < 20000 else torch.from_numpy(np.sort(np.random.default_rng(1).choice(V, 20000, False)))
    paths, (rcp_dt, ext) = ctx.debug_confocal_paths(info, lx, pick.to(cuda))
    ctx.check_device_status()
    paths = paths.cpu().numpy()
    want = numpy_ref.confocal_scatter_given_paths(cube, paths, rcp_dt, ext, info.time_step)
    ok = (paths.astype(np.float64) ** 2 > 2e-5).all(axis=1)
    steps = np.ceil(2 * ext / info.time_step) + 1
    got = got[pick.to(cuda)].cpu().numpy().astype(np.float64)
    assert want[ok].any() and ok.mean() > 0.9
    assert (np.abs(got - want)[ok] <= (32 * steps + 4) * 2.0 ** -24 * want[ok]).all()
