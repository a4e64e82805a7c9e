"""A batch's window stages are cut for one, two or three CTAs to an SM, by the number and the
evenness of its work items; whatever they are, every capture's volume is the single call's, bit
for bit."""
import pytest

pytestmark = pytest.mark.gpu

# (scan side, bins, volume) of each capture: a few items, one or two to an SM, three to an SM in
# one round, more than one round, uneven ones.
BATCHES = {
    "few": [(12, 256, (24, 24, 24))] * 2,
    "two to an SM": [(12, 256, (32, 32, 32))] * 30,
    "three to an SM": [(16, 300, (40, 40, 40))] * 16,
    "more than a round": [(10, 300, (24, 24, 24))] * 64,
    "uneven": [(8 + 4 * (k % 4), 256 + 100 * (k % 3), (24 + k, 40, 32 + (k % 5) * 8)) for k in range(16)],
}


@pytest.mark.parametrize("name", sorted(BATCHES))
def test_batch_equals_single_calls(ctx, cuda, name):
    import torch

    from fasterbackprojection_gb300 import Batch, make_info, scenes

    caps, want = [], []
    made = {}
    for n, T, vres in BATCHES[name]:
        if (n, T, vres) not in made:
            cap = scenes.confocal_points(n, T, 4.92 / T / scenes.LIGHT_SPEED, n_points=30, depth_range=(0.3, 1.3),
                                         seed=n + T)
            hmin, vs = scenes.volume_geometry(vres, depth_range=(0.0, 1.6))
            info = make_info(num_laser_targets=n * n, num_time_bins=T, time_step=cap.time_step, voxel_res=vres,
                             hidden_min=hmin, voxel_size=vs)
            cube, lx = torch.from_numpy(cap.cube).to(cuda), torch.from_numpy(cap.laser_xyz).to(cuda)
            made[(n, T, vres)] = info, cube, lx, ctx.backproject_confocal(info, cube, lx)
        info, cube, lx, vol = made[(n, T, vres)]
        caps.append((info, cube, lx, torch.full_like(vol, float("nan")), 1))
        want.append(vol)
    batch = Batch(ctx, caps)
    batch.run()
    torch.cuda.synchronize()
    ctx.check_device_status()
    batch.close()
    for c, w in zip(caps, want):
        assert float(w.max()) > 0 and torch.equal(c[3], w)
