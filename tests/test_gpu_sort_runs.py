"""GPU: fdf_SortByCell by tiles of ids: both sides of the sizes that choose them, ids of one cell, tiles without a valid
id, spans just below and above the shared counts, runs of equal ids with far jumps between them; a scratch
that stays at a word per cell; and the time of such runs against the way without tiles."""
import ctypes
import time

import numpy as np
import pytest

from tests.test_gpu_sort import reference, sort_by_cell_gpu

pytestmark = pytest.mark.gpu

N = 8 << 20   # from here on a second count instead of ranks
RANKS = 3 << 20   # from here on tiles
TILE, BINS = 8192, 12224


@pytest.mark.parametrize("n,ncells", [(N - 1, 90_000), (N, 90_000), (N + 77, N // 3), (N + 77, N // 3 + 1000), (N + TILE, 700_000),
                                      (RANKS - 1, 40_000), (RANKS + 5, 40_000), (RANKS + TILE, RANKS // 3)])
def test_tiles_of_every_kind(require_gpu, n, ncells):
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
    for k in range(8, 20):                                      # runs that begin and end inside warps
        run = int(rng.integers(2, 90))
        cells[k * t:(k + 1) * t] = np.repeat(rng.integers(0, ncells, t // run + 1), run)[:t]
    cells[rng.random(n) < 0.01] = -1
    cells[-3:] = [ncells, ncells - 1, 0]
    perm, start = sort_by_cell_gpu(cells, ncells)
    ref_perm, ref_start = reference(cells, ncells)
    assert np.array_equal(start, ref_start)
    assert np.array_equal(perm, ref_perm)


def _call(ids, ncells):
    import torch

    from fdf_gb300 import _lib
    lib = _lib.load()
    perm = torch.empty(len(ids), dtype=torch.int32, device="cuda")
    start = torch.empty(ncells + 1, dtype=torch.int32, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    return (lambda: lib.fdf_SortByCell(p(ids), len(ids), ncells, p(perm), p(start), stream)), (perm, start)


def test_scratch_is_a_word_per_cell(require_gpu):
    import torch
    drv = ctypes.CDLL("libcuda.so.1")
    ids = (torch.arange(16_000_000, device="cuda") // 16).to(torch.int32)
    call, keep = _call(ids, 1_000_000)
    pool, used = ctypes.c_void_p(), ctypes.c_uint64(0)
    torch.cuda.synchronize()
    assert drv.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    high = 8   # CU_MEMPOOL_ATTR_USED_MEM_HIGH: set to zero, it starts again from what is in use
    assert drv.cuMemPoolSetAttribute(pool, high, ctypes.byref(used)) == 0
    assert call() == 0
    torch.cuda.synchronize()
    assert drv.cuMemPoolGetAttribute(pool, high, ctypes.byref(used)) == 0
    assert 0 < used.value < 4.5 * 1_000_000


@pytest.mark.parametrize("n", [16_000_000, 6_000_000])
def test_runs_of_equal_ids_with_far_jumps(require_gpu, n):
    """One atomic per id took these twice the time of the way without tiles, one per run of a warp as much (16M: a second
    count; 6M: ranks)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(1)
    ids = torch.randint(0, n // 4, (n // 32,), device="cuda", generator=g).repeat_interleave(32).to(torch.int32).contiguous()
    took = []
    for ncells in (n // 4, n // 3 + 1):   # by tiles, without
        call, keep = _call(ids, ncells)
        best = 1e9
        for _ in range(7):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for _ in range(8):
                assert call() == 0
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t0)
        took.append(best / 8)
    assert took[0] < 1.4 * took[1], took
