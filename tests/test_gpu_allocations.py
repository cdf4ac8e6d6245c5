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


def _fail_one(lib, after):
    assert lib.fdf_TestFailOneDeviceAllocation(int(after)) == 0


@pytest.fixture
def holding():
    """A context that holds the buffer of a points call."""
    coor = W.sinusoidal_grid(6, 5, 8, amp=0.02)
    with PicContext(0) as ctx:
        ctx.set_grid(coor)
        ctx.set_ucat(np.ones((8, 5, 6, 3)))
        pos, cell = W.volumetric_particles(coor, 50_000, seed=2)
        want = ctx.locate_points(pos, cell)
        yield ctx, pos, cell, want
        _fail_one(ctx.lib, -1)


def test_a_kept_buffer_gives_way(holding):
    """An allocation that finds no room takes the buffer that a points call left, where it was refused before."""
    ctx, pos, cell, want = holding
    n = 5_000_000   # more than the context keeps: the call's own buffer
    many = np.resize(pos, (n, 3)), np.resize(cell, (n, 3))
    calls = [lambda: ctx.locator_init(1), lambda: ctx.set_momentum_deposit(True),
             lambda: ctx.set_ucont(np.zeros((9, 6, 7, 3))), lambda: ctx.grid_metrics(), lambda: ctx.locate_points(*many)]
    for call in calls:
        ctx.locate_points(pos, cell)
        _fail_one(ctx.lib, 0)
        call()
        got = ctx.locate_points(pos, cell)
        for a, b in zip(got, want):
            assert np.array_equal(a, b)


def test_a_buffer_in_use_stays(holding):
    """Training's scratch finds no room while the call's samples lie in the kept buffer: the call is refused, the next
    one works."""
    ctx, pos, cell, want = holding
    ctx.locator_init(1)
    _fail_one(ctx.lib, 0)   # (the samples fit in the kept buffer: the scratch is the first allocation)
    with pytest.raises(PetscError) as e:
        ctx.locator_train(1000, seed=1, steps=3, batch=4096)
    assert e.value.code == 55
    assert np.isfinite(ctx.locator_train(1000, seed=1, steps=3, batch=4096)).all()
    for a, b in zip(ctx.locate_points(pos, cell), want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n,ncells", [(1000, 77), (70_000, 9000)])
def test_sort_without_room_for_ranks(require_gpu, n, ncells):
    from fdf_gb300 import _lib
    from tests.test_gpu_sort import reference, sort_by_cell_gpu
    lib = _lib.load()
    cells = np.random.default_rng(n).integers(-5, ncells + 5, n)
    _fail_one(lib, 0)
    try:
        perm, start = sort_by_cell_gpu(cells, ncells)
    finally:
        _fail_one(lib, -1)
    ref_perm, ref_start = reference(cells, ncells)
    assert np.array_equal(start, ref_start) and np.array_equal(perm, ref_perm)
