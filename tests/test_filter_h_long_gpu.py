"""filter_H on long series: on both sides of the lengths where the rows of a series in shared
memory change their form (some 6,000 and 11,000 bins at the default wavelength), up to the
longest that one CTA can hold, and just above it; and short series with many taps.

The bound is the one of the launch shapes: (taps + 2) 2^-24 sum |tap| |sample|."""
import numpy as np
import pytest

from tests import test_filter_h_sizes_gpu as sizes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("border", ["zero", "edge"])
@pytest.mark.parametrize("n,T,wl_bins", [(3, 6000, 10.0), (3, 6040, 10.0), (400, 8191, 4.0), (2, 11040, 10.0),
                                         (700, 11104, 10.0), (2, 38500, 10.0), (1, 57774, 10.0), (3, 45000, 4.0),
                                         (2, 20000, 30.0), (2, 45000, 60.0), (5, 128, 150.0), (3, 2500, 40.0)])
def test_long_series_vs_fp64(ctx, cuda, n, T, wl_bins, border):
    sizes.test_filter_h_launch_shapes_vs_fp64(ctx, cuda, n, T, wl_bins, border)


def test_longer_series_are_refused(ctx, cuda):
    import torch

    from fasterbackprojection_gb300._lib import FbpError

    with pytest.raises(FbpError, match="too long"):
        ctx.filter_h_(torch.zeros((1, 57775), device=cuda), 0.0048, wl_mean=0.048)
