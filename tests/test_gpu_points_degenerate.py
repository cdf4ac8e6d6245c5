"""GPU: points located in grids with and without a degenerate cell, one grid after another in the same context."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import PetscError, PicContext

pytestmark = pytest.mark.gpu


def test_degenerate_cells_and_then_none(require_gpu):
    good = W.uniform_grid(2, 1, 1)
    bad = good.copy()
    bad[:, :, 0, :] = bad[:, :, 1, :]           # the first cell has no width
    point = np.array([[0.75, 0.5, 0.5]])
    there = np.array([[1, 0, 0]])
    with PicContext(0) as ctx:
        for grid in (bad, good, bad, bad, good):
            ctx.set_grid(grid)
            for _ in range(2):
                if grid is bad:
                    with pytest.raises(PetscError) as e:
                        ctx.locate_points(point)            # from cell (0,0,0)
                    assert e.value.code == 83
                else:
                    cell, _, status = ctx.locate_points(point)
                    assert np.array_equal(cell, there) and status[0] == 1
                cell, _, status = ctx.locate_points(point, there)   # a walk that meets the good cell only
                assert np.array_equal(cell, there) and status[0] == 1
