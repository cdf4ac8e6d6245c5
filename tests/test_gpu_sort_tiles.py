"""GPU: fdf_SortByCell where blocks of ids nearly in order count them in shared memory: both sides of the sizes that
choose it, ids of one cell, blocks with no valid id, spans just below and above the shared counts, and
blocks of both kinds in one call."""
import numpy as np
import pytest

from tests.test_gpu_sort import reference, sort_by_cell_gpu

pytestmark = pytest.mark.gpu

N = 3 << 20
TILE, BINS = 8192, 12224


@pytest.mark.parametrize("n,ncells", [(N - 1, 50_000), (N, 50_000), (N + 77, N // 3), (N + 77, N // 3 + 1000), (N + TILE, 400_000)])
def test_nearly_sorted_ids(require_gpu, n, ncells):
    rng = np.random.default_rng(n + ncells)
    cells = np.arange(n, dtype=np.int64) * ncells // n + rng.integers(-500, 501, n)   # some below zero or past the last
    t = TILE
    cells[0:t] = 17                                       # one cell
    cells[t:2 * t] = -1                                   # none
    cells[3 * t:4 * t] = rng.integers(100, 100 + BINS, t)       # as many cells as there are counts
    cells[3 * t], cells[3 * t + 1] = 100, 100 + BINS - 1
    cells[4 * t:5 * t] = rng.integers(100, 100 + BINS, t)
    cells[4 * t], cells[4 * t + 1] = 100, 100 + BINS            # one more
    cells[5 * t:6 * t] = rng.integers(0, ncells, t)             # the whole range
    cells[6 * t + 5] = ncells - 1                               # an outlier
    cells[rng.random(n) < 0.01] = -1
    cells[-3:] = [ncells, ncells - 1, 0]
    perm, start = sort_by_cell_gpu(cells, ncells)
    ref_perm, ref_start = reference(cells, ncells)
    assert np.array_equal(start, ref_start)
    assert np.array_equal(perm, ref_perm)
