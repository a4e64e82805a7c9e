"""The sums of a gather's chains ask for 128 MB at most, and the buffers that a context has
outgrown (kept for graphs captured with them) are bounded with the current one by twice that."""
import pytest

from tests.test_gather_chains_gpu import _capture

pytestmark = pytest.mark.gpu


def test_outgrown_buffers_are_bounded(cuda):
    import torch

    from fasterbackprojection_gb300 import Context

    ctx = Context()
    # 60, 80 and 128 MB of sums, after rows that are the longest and leave no room behind them.
    calls = [_capture(cuda, n, T, v, 1) for n, T, v in ((64, 1024, (256, 256, 256)), (32, 256, (96, 128, 160)),
                                                        (64, 512, (128, 128, 80)), (64, 512, (128, 128, 128)))]
    outs = [torch.empty(tuple(c[0].voxel_res)[::-1], device=cuda) for c in calls]
    ctx.backproject_confocal(*calls[0], out=outs[0])
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for c, o in zip(calls[1:], outs[1:]):
        before = ctx.launches
        ctx.backproject_confocal(*c, out=o)
        assert ctx.launches - before == 3  # in several chains
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    ctx.check_device_status()
    ctx.close()
    assert 128 << 20 <= used <= (256 << 20) + (4 << 20)
