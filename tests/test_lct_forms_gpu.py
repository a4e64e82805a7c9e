"""The fused LCT where its launches change form: short lines with few and with many CTAs, every
line length up to 4096, both orders of the capture, and inputs and outputs that start one element
past an aligned address.

Against the FP64 restatement to 1e-5 relative L2: two three-dimensional transforms and the PSF's,
at most 26 stages each of one rounding (2^-24), 78 * 6e-8 = 4.7e-6 in the worst case, and the two
resamplings.  The forms of one size give the same bits."""
import numpy as np
import pytest

from oracle import numpy_ref
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(8, 16), (16, 32), (32, 64), (64, 64), (64, 128), (128, 16), (128, 32), (8, 128),
                                 (8, 256), (16, 512), (8, 1024), (8, 2048)])
def test_lct_forms(ctx, cuda, n, m):
    import torch
    from fasterbackprojection_gb300 import FBP_LAYOUT_TIME_INNER, FBP_LAYOUT_TIME_MAJOR

    rng = np.random.default_rng(n * m)
    data = rng.poisson(rng.uniform(0, 20, (m, n, n))).astype(np.float32)  # [M][N][N]
    step = 4.92 / m
    want = numpy_ref.lct(data.astype(np.float64), 1.0, step, 0.8, True)
    first = None
    for layout in (FBP_LAYOUT_TIME_MAJOR, FBP_LAYOUT_TIME_INNER):
        host = data if layout == FBP_LAYOUT_TIME_MAJOR else np.ascontiguousarray(data.transpose(1, 2, 0))
        for shift in (0, 1):
            src = torch.empty(data.size + 4, device=cuda)[shift:shift + data.size].view(*host.shape)
            src.copy_(torch.from_numpy(host))
            out = torch.full((data.size + 4,), float("nan"), device=cuda)[shift:shift + data.size].view(m, n, n)
            ctx.lct(src, 1.0, step, 0.8, True, layout=layout, out=out)
            if first is None:
                first = out.clone()
                assert rel_l2(first.cpu().numpy(), want) < 1e-5
            assert torch.equal(out, first), (layout, shift)


@pytest.mark.parametrize("n", [1, 3, 1023, 4097, 1000003])
def test_normalise_off_alignment(ctx, cuda, n):
    import torch

    v = torch.rand(n, generator=torch.Generator().manual_seed(n)).to(cuda)
    want = ctx.normalize_(v.clone())
    for shift in (1, 2, 3):
        w = torch.empty(n + 4, device=cuda)[shift:shift + n]
        w.copy_(v)
        assert torch.equal(ctx.normalize_(w), want)
