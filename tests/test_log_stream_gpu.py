"""The streaming LoG filter at the edges of its tiles (32 x 8 columns, runs of 8
planes and more), against the FP64 oracle on the same taps.

Bound per voxel, from the rounding of a sum of k^3 fused products:
(k^3 + 2) 2^-24 sum |tap| |sample|; it holds where the taps cancel (a volume of
one voxel is nothing but border)."""
import numpy as np
import pytest

from oracle import cpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 5), (8, 8, 32), (9, 9, 33), (17, 7, 31), (65, 16, 48), (130, 20, 16),
                                   (3, 40, 70)])
@pytest.mark.parametrize("ksize,sigma", [(3, 0.8), (5, 1.0)])
def test_log_stream_vs_oracle(ctx, cuda, shape, ksize, sigma):
    import torch
    from fasterbackprojection_gb300 import FBP_FILTER_LOG

    rng = np.random.default_rng(sum(shape) + ksize)
    v = rng.standard_normal(shape).astype(np.float32)
    got = ctx.postfilter(FBP_FILTER_LOG, torch.from_numpy(v).to(cuda), ksize, sigma).cpu().numpy().astype(np.float64)
    w = cpu.log_weights(ksize, sigma)
    want = cpu.log_filter(v, w, ksize)
    size = cpu.log_filter(np.abs(v), np.abs(w), ksize)
    assert (np.abs(got - want) <= (ksize ** 3 + 2) * 2.0 ** -24 * size).all()
