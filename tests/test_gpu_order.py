"""GPU: the order within a cell and within the LOST particles, at the sizes where the sort changes hands."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import FORM_FP32, FORM_PLAIN_FP64, LOST, PicContext, SwarmArrays
from tests.test_gpu_sort import reference, sort_by_cell_gpu

pytestmark = pytest.mark.gpu


def test_cell_lengths_across_the_thresholds(require_gpu):
    """Cells of 0 to 1100 slots in one array: thread, lanes, warp, block in shared memory, block in place."""
    lengths = [7, 8, 9, 16, 16, 17, 31, 32, 33, 64, 127, 128, 129, 1023, 1024, 1025, 1100, 0, 1, 2, 40, 40, 9, 130]
    rng = np.random.default_rng(3)
    cells = np.repeat(np.arange(len(lengths)) * 3, lengths)
    rng.shuffle(cells)
    ncells = 3 * len(lengths)
    perm, start = sort_by_cell_gpu(cells, ncells)
    ref_perm, ref_start = reference(cells, ncells)
    assert np.array_equal(start, ref_start)
    assert np.array_equal(perm, ref_perm)


@pytest.mark.parametrize("form", [FORM_PLAIN_FP64, FORM_FP32])
@pytest.mark.parametrize("lost", [0, 1, 2047, 2048, 2049, 4097, 70_001])
def test_lost_particles_keep_their_order(require_gpu, form, lost):
    """The initial setup keeps the LOST particles behind the located ones: by PID in the plain form,
    in their previous order in the precision form; crowded cells (50 per cell) likewise."""
    coor = W.uniform_grid(4, 4, 4)
    rng = np.random.default_rng(lost + 1)
    n_in = 3200
    pos = np.concatenate([rng.uniform(0.02, 0.98, (n_in, 3)), rng.uniform(2.0, 3.0, (lost, 3))])
    shuffle = rng.permutation(len(pos))
    pos, pid = pos[shuffle], rng.permutation(len(pos)).astype(np.int64)
    with PicContext(0) as ctx:
        ctx.set_form(form)
        ctx.set_grid(coor)
        ctx.set_ucat(np.zeros((4, 4, 4, 3)))
        ctx.set_dt(0.0)
        ctx.set_swarm(SwarmArrays.create(pos, pid=pid))
        ctx.initial_setup()
        s = ctx.get_swarm()
    assert s.n == len(pos)
    gone = s.status == LOST
    assert gone.sum() == lost and np.all(gone[n_in:])
    slot = np.empty(len(pos), dtype=np.int64)
    slot[pid] = np.arange(len(pos))
    key = s.pid if form == FORM_PLAIN_FP64 else slot[s.pid]
    cell = (s.cell[:, 2] * 4 + s.cell[:, 1]) * 4 + s.cell[:, 0]
    cell[gone] = 64
    assert np.array_equal(np.lexsort((key, cell)), np.arange(len(pos)))
