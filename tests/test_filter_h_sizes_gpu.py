"""filter_H at the edges of its launch shapes: series of up to 256, 512 and more
bins take 32, 64 and 128 threads, series with more slots than a thread keeps
load the rest in a second way, and few series give each CTA less than one.

Bound per bin, from the rounding of a sum of m products (each tap and each
product-sum step rounds once): (m + 2) 2^-24 sum |tap| |sample|, with m the taps
the kernel keeps.  It holds whatever cancels in the band-pass."""
import numpy as np
import pytest

from oracle import numpy_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("border", ["zero", "edge"])
@pytest.mark.parametrize("n,T,wl_bins", [(1, 1, 3.0), (3, 255, 10.0), (2000, 256, 4.0), (5, 257, 16.0), (700, 511, 10.0),
                                         (9, 513, 10.0), (40, 1025, 6.0), (3, 1500, 12.0), (7, 2048, 20.0)])
def test_filter_h_launch_shapes_vs_fp64(ctx, cuda, n, T, wl_bins, border):
    import torch

    rng = np.random.default_rng(T)
    data = rng.poisson(rng.uniform(0, 40, (n, T))).astype(np.float32)
    dt = 0.0048
    wl = dt * wl_bins
    got = ctx.filter_h_(torch.from_numpy(data.copy()).to(cuda), dt, wl_mean=wl,
                        border=1 if border == "edge" else 0).cpu().numpy().astype(np.float64)
    pick = rng.choice(n, min(n, 20), replace=False)
    want = numpy_ref.filter_h(data[pick], dt, wl_mean=wl, border=border)
    # sum |tap| |sample|: the same circular convolution with the taps' magnitudes.
    sigma, t6, npad = numpy_ref.filter_h_params(T, dt, wl)
    K = numpy_ref.filter_h_kernel(npad, float(np.float32(dt)), float(np.float32(wl)), sigma)
    pad = (npad - T) // 2
    x = np.pad(data[pick].astype(np.float64), ((0, 0), (pad, npad - T - pad)),
               **({"mode": "edge"} if border == "edge" else {"mode": "constant"}))
    taps = npad * np.abs(K.real)
    size = np.fft.irfft(np.fft.rfft(x) * np.fft.rfft(taps)[None], n=npad)[:, pad:pad + T]
    m = int((taps > 1e-12 * taps.max()).sum())
    assert (np.abs(got[pick] - want) <= (m + 2) * 2.0 ** -24 * size + 1e-30).all()
