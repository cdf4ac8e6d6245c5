"""GPU: how many device allocations a grid takes, counted by letting the one after them fail on the host."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import PetscError, PicContext

pytestmark = pytest.mark.gpu


def _fail_allocations(lib, after):
    assert lib.fdf_TestFailDeviceAllocations(int(after)) == 0


def test_a_grid_takes_nineteen_allocations(require_gpu):
    coor = W.uniform_grid(5, 4, 3)
    with PicContext(0) as ctx:
        for budget in (18, 19):
            _fail_allocations(ctx.lib, budget)
            try:
                if budget < 19:
                    with pytest.raises(PetscError):
                        ctx.set_grid(coor)
                else:
                    ctx.set_grid(coor)
            finally:
                _fail_allocations(ctx.lib, -1)
        ctx.set_ucat(np.zeros((3, 4, 5, 3)))
        ctx.seed_particles(100, 1)
        assert ctx.initial_setup().n_end == 100
