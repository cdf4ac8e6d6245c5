"""GPU: the ordering of the particles without a cell is one launch whatever the capacity, and its merges across the
blocks give the same order call after call, for lengths of two to many chunks, in both forms."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import FORM_FP32, FORM_PLAIN_FP64, LOST, PicContext, SwarmArrays

pytestmark = pytest.mark.gpu


def _context(form, pos, pid, room):
    ctx = PicContext(0)
    ctx.set_form(form)
    ctx.set_grid(W.uniform_grid(4, 4, 4))
    ctx.set_ucat(np.zeros((4, 4, 4, 3)))
    ctx.set_dt(0.0)
    ctx.reserve(room)
    ctx.set_swarm(SwarmArrays.create(pos, pid=pid))
    return ctx


@pytest.mark.parametrize("form", [FORM_PLAIN_FP64, FORM_FP32])
def test_launches_do_not_grow_with_the_capacity(require_gpu, form):
    pos = np.random.default_rng(1).uniform(0.02, 0.98, (1000, 3))
    made = []
    for room in (1000, 3_000_000):
        with _context(form, pos, np.arange(1000), room) as ctx:
            ctx.initial_setup()
            k = []
            for call in (ctx.initial_setup, ctx.locate, ctx.remove_lost, ctx.remove_out_of_bounds):
                before = ctx.launches
                call()
                k.append(ctx.launches - before)
            made.append(k)
    assert made[0] == made[1]
    assert max(made[1]) <= 9


@pytest.mark.parametrize("form", [FORM_PLAIN_FP64, FORM_FP32])
@pytest.mark.parametrize("lost", [2 * 2048 + 1, 3 * 2048, 8 * 2048, 8 * 2048 + 1, 400_000])
def test_many_chunks_again_and_again(require_gpu, form, lost):
    rng = np.random.default_rng(lost)
    n_in = 500
    pos = np.concatenate([rng.uniform(0.02, 0.98, (n_in, 3)), rng.uniform(2.0, 3.0, (lost, 3))])
    pos = pos[rng.permutation(len(pos))]
    pid = rng.permutation(len(pos)).astype(np.int64)
    with _context(form, pos, pid, 2 * len(pos)) as ctx:
        ctx.initial_setup()
        first = ctx.get_swarm()
        for _ in range(6):
            ctx.reset_statuses()
            ctx.locate()
        again = ctx.get_swarm()
    gone = first.status == LOST
    assert gone.sum() == lost and np.all(gone[n_in:])
    where = np.empty(len(pos), dtype=np.int64)
    where[pid] = np.arange(len(pos))
    key = first.pid if form == FORM_PLAIN_FP64 else where[first.pid]
    cell = (first.cell[:, 2] * 4 + first.cell[:, 1]) * 4 + first.cell[:, 0]
    cell[gone] = 64
    assert np.array_equal(np.lexsort((key, cell)), np.arange(len(pos)))
    assert np.array_equal(first.pid, again.pid) and np.array_equal(first.cell, again.cell)
