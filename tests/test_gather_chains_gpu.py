"""The gathers' chains: small volumes split the scan points (or pairs) of a voxel
tile over several CTAs (1 to 32 chains), each with its own compensated sums.

  * against the FP64 oracle with the GPU's bins: 1e-6 relative L2, the bound of
    the unsplit gather (FP32 sums of at most 32 terms and compensated folds:
    32 * 2^-24 / 2 = 9.5e-7 for the worst case, far less in practice);
  * a batch walks the same chains one after the other in one CTA: bit for bit.
"""
import numpy as np
import pytest

from oracle import cpu
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

# scan side, bins, volume, bounces kept, time offset.  Groups of 32 scan points:
# 1, 2, 3, 5, 8 and 13 of them, the last one ragged; volumes of one voxel, one
# tile, one tile plus a row on each axis, and with idle warps; windows that
# are the whole row (few bins per voxel) and that are not.
CASES = [
    (3, 64, (1, 1, 1), False, 0.0),
    (5, 128, (16, 16, 16), False, 0.0),
    (8, 512, (17, 17, 17), False, 0.0),
    (9, 96, (33, 9, 5), True, 0.0),
    (12, 512, (40, 33, 17), True, 0.4),
    (16, 640, (48, 20, 36), False, 0.4),
    (20, 300, (16, 64, 24), True, -0.1),
    (20, 2048, (21, 24, 40), False, 0.0),
]


@pytest.mark.parametrize("n,T,vres,bounce,t0", CASES)
def test_chains_against_fp64_and_against_the_batch(ctx, cuda, n, T, vres, bounce, t0):
    import torch

    from fasterbackprojection_gb300 import Batch, make_info, scenes

    cap = scenes.confocal_points(n, T, 4.92 / T / scenes.LIGHT_SPEED, n_points=40, depth_range=(0.3, 1.3), seed=n + T)
    hmin, vs = scenes.volume_geometry(vres, depth_range=(0.0, 1.6))
    info = make_info(num_laser_targets=n * n, num_time_bins=T, time_step=cap.time_step, voxel_res=vres,
                     hidden_min=hmin, voxel_size=vs, discard_first_last_bounces=0 if bounce else 1, time_offset=t0,
                     laser_position=(0.05, -0.25, 0.1), sensor_position=(-0.1, -0.2, 0.05))
    cube = torch.from_numpy(cap.cube).to(cuda)
    lx = torch.from_numpy(cap.laser_xyz).to(cuda)
    vol = ctx.backproject_confocal(info, cube, lx)
    bins = ctx.debug_confocal_bins(info, lx, torch.arange(vol.numel(), device=cuda)).cpu().numpy()
    again = torch.full_like(vol, float("nan"))
    batch = Batch(ctx, [(info, cube, lx, again, 1)])
    batch.run()
    torch.cuda.synchronize()
    ctx.check_device_status()
    batch.close()
    want = cpu.confocal_voxel(info, cap.cube, cap.laser_xyz, bins=bins)
    assert (bins >= 0).any()
    assert rel_l2(vol.cpu().numpy(), want) < 1e-6
    assert torch.equal(vol, again)


# laser side, SPAD side, bins, volume, bounces kept, time offset: laser blocks
# of 4 that are whole (4, 16, 36 lasers), padded (9, 25) or not taken (1), pair
# groups of 32 that are one, ragged or many, volumes of one voxel, one tile and
# one tile plus a row; windows that are the whole row; paths around zero.
EXHAUSTIVE = [
    (1, 1, 64, (1, 1, 1), False, 0.0),
    (2, 3, 96, (8, 16, 16), True, 0.0),
    (1, 6, 512, (9, 17, 17), False, 0.0),
    (3, 5, 300, (17, 9, 5), False, 0.5),
    (3, 7, 1024, (24, 20, 36), True, 0.5),
    (4, 6, 256, (16, 33, 20), False, -0.3),
    (5, 4, 2048, (21, 16, 16), False, 0.0),
    (6, 9, 640, (40, 24, 24), True, -0.2),
]


@pytest.mark.parametrize("nl,ns,T,vres,bounce,t0", EXHAUSTIVE)
def test_exhaustive_chains_against_fp64(ctx, cuda, nl, ns, T, vres, bounce, t0):
    import torch

    from fasterbackprojection_gb300 import FBP_EXHAUSTIVE, make_info, scenes

    cap = scenes.exhaustive_points(nl, ns, T, 4.92 / T / scenes.LIGHT_SPEED, n_points=40, depth_range=(0.3, 1.3),
                                   seed=nl + T)
    hmin, vs = scenes.volume_geometry(vres, depth_range=(0.0, 1.6))
    info = make_info(num_laser_targets=nl * nl, num_sensor_targets=ns * ns, num_time_bins=T, time_step=cap.time_step,
                     voxel_res=vres, hidden_min=hmin, voxel_size=vs, capture_system=FBP_EXHAUSTIVE,
                     discard_first_last_bounces=0 if bounce else 1, time_offset=t0,
                     laser_position=(0.05, -0.25, 0.1), sensor_position=(-0.1, -0.2, 0.05))
    lx = torch.from_numpy(cap.laser_xyz).to(cuda)
    sx = torch.from_numpy(cap.sensor_xyz).to(cuda)
    vol = ctx.backproject_exhaustive(info, torch.from_numpy(cap.cube).to(cuda), lx, sx)
    bins = ctx.debug_exhaustive_bins(info, lx, sx, torch.arange(vol.numel(), device=cuda)).cpu().numpy()
    ctx.check_device_status()
    want = cpu.exhaustive_voxel(info, cap.cube, cap.laser_xyz, cap.sensor_xyz, bins=bins)
    assert (bins >= 0).any()
    assert rel_l2(vol.cpu().numpy(), want) < 1e-6


def _capture(cuda, n, T, vres, seed):
    import torch

    from fasterbackprojection_gb300 import make_info, scenes

    cap = scenes.confocal_points(n, T, 4.92 / T / scenes.LIGHT_SPEED, n_points=20, depth_range=(0.3, 1.3), seed=seed)
    hmin, vs = scenes.volume_geometry(vres, depth_range=(0.0, 1.6))
    info = make_info(num_laser_targets=n * n, num_time_bins=T, time_step=cap.time_step, voxel_res=vres,
                     hidden_min=hmin, voxel_size=vs, discard_first_last_bounces=1)
    return info, torch.from_numpy(cap.cube).to(cuda), torch.from_numpy(cap.laser_xyz).to(cuda)


def _launches(ctx, call):
    before = ctx.launches
    out = call()
    return ctx.launches - before, out


@pytest.fixture()
def own_ctx(cuda):
    from fasterbackprojection_gb300 import Context

    c = Context()
    yield c
    c.check_device_status()
    c.close()


def test_capture_without_chain_scratch_runs_one_chain(own_ctx, cuda):
    """A context that has only run a volume too large for chains can be captured
    with a smaller one, although its chains' sums would need an allocation: one
    CTA per tile then, the same volume to FP32 rounding."""
    import torch

    ctx = own_ctx
    big = _capture(cuda, 32, 1024, (256, 256, 256), 1)  # rows and tables as large as the small one needs
    small = _capture(cuda, 32, 256, (32, 32, 32), 2)
    assert _launches(ctx, lambda: ctx.backproject_confocal(*big))[0] == 2  # rows, gather
    out = torch.empty((32, 32, 32), device=cuda)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        count, _ = _launches(ctx, lambda: ctx.backproject_confocal(*small, out=out))
    assert count == 2
    graph.replay()
    count, eager = _launches(ctx, lambda: ctx.backproject_confocal(*small))
    assert count == 3  # the chains' fold too
    assert rel_l2(out.cpu().numpy(), eager.cpu().numpy()) < 1e-6


def test_captured_chains_outlive_a_call_that_needs_more(own_ctx, cuda):
    """A captured call keeps its chain scratch when a later call with fewer scan
    points, but more voxels, outgrows it."""
    import torch

    ctx = own_ctx
    first = _capture(cuda, 32, 512, (16, 16, 170), 3)
    more = _capture(cuda, 20, 256, (64, 64, 72), 4)
    ctx.backproject_confocal(*_capture(cuda, 32, 2048, (256, 256, 256), 5))  # rows without room for sums behind them
    want = ctx.backproject_confocal(*first)
    out = torch.empty_like(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.backproject_confocal(*first, out=out)
    again = ctx.backproject_confocal(*more)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert torch.equal(ctx.backproject_confocal(*more), again)
