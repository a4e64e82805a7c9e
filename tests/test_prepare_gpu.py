"""The gathers' rows at the edges of the launch that makes them: captures of one
sample, of bins that are and are not a multiple of four, aligned and not, in
both layouts and every storage type, all give the volume of the same samples in
FP32, time innermost, bit for bit; samples at and below the threshold, negative
ones and NaN count as zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,T", [(1, 1), (1, 4), (3, 31), (6, 33), (7, 64), (16, 510), (33, 1024)])
def test_rows_of_every_form_agree_bitwise(ctx, cuda, n, T):
    import torch

    from fasterbackprojection_gb300 import (FBP_LAYOUT_TIME_INNER, FBP_LAYOUT_TIME_MAJOR, make_info, scenes)

    L = n * n
    rng = np.random.default_rng(100 * n + T)
    hmin, vs = scenes.volume_geometry((9, 10, 11), depth_range=(0.0, 1.6))
    info = make_info(num_laser_targets=L, num_time_bins=T, time_step=5.0 / T, voxel_res=(9, 10, 11), hidden_min=hmin,
                     voxel_size=vs, discard_first_last_bounces=1)
    lx = torch.from_numpy(rng.uniform(-1, 1, (L, 3)).astype(np.float32)).to(cuda)
    lx[:, 1] = 0
    dirty = torch.from_numpy(rng.integers(1, 200, (L, T)).astype(np.float32)).to(cuda)
    drop = torch.from_numpy(rng.integers(0, 4, (L, T))).to(cuda)
    dirty[drop == 0] = torch.tensor([0.0, -3.0, 1e-5, float("nan")], device=cuda).repeat(L * T)[: int((drop == 0).sum())]
    eps = torch.tensor(1e-5, device=cuda)
    for dtype in (torch.float32, torch.bfloat16, torch.float16):
        stored = dirty.to(dtype).float()  # 1e-5 rounds up in bf16: a sample that counts
        want = ctx.backproject_confocal(info, torch.where(stored > eps, stored, torch.zeros_like(stored)), lx)
        assert T < 16 or float(want.max()) > 0
        for layout in (FBP_LAYOUT_TIME_INNER, FBP_LAYOUT_TIME_MAJOR):
            cube = (dirty if layout == FBP_LAYOUT_TIME_INNER else dirty.t().contiguous()).to(dtype)
            for shift in (0, 1):  # one element past an aligned start
                buf = torch.zeros(L * T + 4, dtype=dtype, device=cuda)
                view = buf[shift: shift + L * T]
                view.copy_(cube.view(-1))
                got = ctx.backproject_confocal(info, view, lx, layout=layout)
                assert torch.equal(want, got), (dtype, layout, shift)
    ctx.check_device_status()
