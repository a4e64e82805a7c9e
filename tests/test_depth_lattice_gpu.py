"""Depth planes behind a regular flat wall, where a tile's threads take its columns: several
tiles and ragged ones (17, 18 and 33 points a side), windows that are the whole row, paths around
zero, a grid of which only some tiles are regular.  Against the kernel that reads the rows from
global memory: the same bins, FP32 sums in another order, 1e-6 relative L2."""
import numpy as np
import pytest

from tests.conftest import rel_l2
from tests.test_depth_tiles_gpu import _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("displaced", [False, True])
@pytest.mark.parametrize("T,bounce,t0", [(96, False, 0.0), (96, True, 0.0), (700, False, 0.0), (700, False, 0.7),
                                         (700, False, -0.3), (700, True, 0.7), (2048, False, 0.0), (2048, False, 0.7)])
@pytest.mark.parametrize("side", [17, 18, 33])
def test_lattice_equals_the_row_kernel(ctx, cuda, side, T, bounce, t0, displaced):
    rng = np.random.default_rng(side + T)
    L = side * side
    gx, gz = np.meshgrid(np.linspace(-1, 1, side), np.linspace(-1, 1, side))
    xyz = np.stack([gx.ravel(), np.full(L, 0.01), gz.ravel()], axis=1).astype(np.float32)
    if displaced:
        xyz[side + 3] += np.float32([0.01, 0.002, -0.01])  # in the first tile
    cube = rng.poisson(3.0, (L, T)).astype(np.float32)
    cube[rng.random((L, T)) < 0.3] = 5e-6  # at or below the threshold: skipped
    got, want = _pair(ctx, cuda, L, T, rng.uniform(0.0, 1.2, 17), (0, -1, 0), bounce, t0, side % 2, xyz, cube)
    assert want.any()
    assert rel_l2(got, want) < 1e-6
