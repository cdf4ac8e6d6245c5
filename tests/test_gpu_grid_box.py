"""GPU: the grid's bounding box with its least and greatest coordinates at each of the first and last nodes, for even and
odd numbers of nodes, read through the locator's normalisation (its centre and half width)."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import PicContext

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 2, 2), (3, 2, 2), (1, 1, 1), (4, 4, 6)])
def test_extremes_anywhere(require_gpu, dims):
    with PicContext(0) as ctx:
        for at in (0, 1, 2, -3, -2, -1):
            for sign in (1.0, -1.0):
                coor = W.uniform_grid(*dims)
                coor.reshape(-1, 3)[at] += sign * np.array([0.11, 0.23, 0.37])
                ctx.set_grid(coor)
                lo, hi = coor.reshape(-1, 3).min(0) - 1e-6, coor.reshape(-1, 3).max(0) + 1e-6
                centre, inv_half = ctx.locator_normalization()
                assert np.array_equal(centre, (0.5 * (lo + hi)).astype(np.float32))
                assert np.array_equal(inv_half, (2.0 / (hi - lo)).astype(np.float32))
