"""Depth planes at a non-finite depth: 0 * depth makes that plane's points NaN (int(NaN) is
bin 0, like the reference's cast) and no other plane's, wherever it stands in a block of
16 planes; the last place, which also stands in for the planes beyond the end, included.
Against the kernel that reads the rows from global memory, to 1e-6 relative L2."""
import numpy as np
import pytest

from tests.conftest import rel_l2
from tests.test_depth_tiles_gpu import _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,flat", [(17, True), (17, False)])
@pytest.mark.parametrize("D,at", [(1, 0), (3, 2), (5, 0), (16, 15), (20, 15), (20, 19)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_a_non_finite_depth_stays_in_its_plane(ctx, cuda, side, flat, D, at, value):
    rng = np.random.default_rng(D + at)
    L, T = side * side, 256
    gx, gz = np.meshgrid(np.linspace(-1, 1, side), np.linspace(-1, 1, side))
    y = np.zeros(L) if flat else rng.uniform(-0.01, 0.01, L)
    xyz = np.stack([gx.ravel(), y, gz.ravel()], axis=1).astype(np.float32)
    depths = np.linspace(0.3, 1.2, D)
    depths[at] = value
    cube = rng.poisson(3.0, (L, T)).astype(np.float32)
    got, want = _pair(ctx, cuda, L, T, depths, (0, -1, 0), False, 0.0, 1, xyz, cube)
    assert want.any()
    for d in range(D):
        assert rel_l2(got[:, d], want[:, d]) < 1e-6, d
