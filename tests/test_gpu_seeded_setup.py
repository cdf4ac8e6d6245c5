"""GPU: the first sort of a seeded swarm, on both sides of the particle count from which it gathers packed
records: the same bits as the setup of the same particles handed over by the caller, which never packs."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import FORM_FP32, FORM_PLAIN_FP64, PicContext

pytestmark = pytest.mark.gpu

LINE = 3 << 19
FIELDS = ("position", "velocity", "weight", "P", "cell", "pid", "status")


def state(ctx):
    s = ctx.get_swarm()
    return [getattr(s, f) for f in FIELDS] + list(ctx.get_scattered()) + list(ctx.get_faces())


def same(a, b, what):
    assert len(a) == len(b)
    for q, (x, y) in enumerate(zip(a, b)):
        assert np.array_equal(x.view(np.int64), y.view(np.int64)), (what, q)


@pytest.mark.parametrize("form", [FORM_PLAIN_FP64, FORM_FP32])
@pytest.mark.parametrize("n", [LINE - 1, LINE, LINE + 257])
def test_setup_of_a_seeded_swarm(require_gpu, form, n):
    IM, JM, KM = 13, 11, 40
    coor = W.bent_pipe_grid(IM, JM, KM)
    ucat = W.field_pipe(coor, W.cell_centroids(coor))
    with PicContext(0) as ctx:
        ctx.set_grid(coor)
        ctx.set_ucat(ucat)
        ctx.set_dt(1e-3)
        ctx.set_form(form)
        ctx.reserve(n + 1000)   # slots beyond the swarm
        ctx.seed_particles(n, seed=3, pid_base=1 << 40, start_in_generating_cell=False)
        held = ctx.get_swarm()
        ctx.initial_setup()
        got = state(ctx)
        ctx.step()
        after = state(ctx)
        ctx.initial_setup()     # of a sorted swarm
        again = state(ctx)
        ctx.set_swarm(held)
        ctx.initial_setup()
        same(got, state(ctx), "setup")
        ctx.step()
        same(after, state(ctx), "step")
        ctx.initial_setup()
        same(again, state(ctx), "second setup")
        # seeded, sorted by the location alone, then set up; and seeded, then stepped at once
        ctx.seed_particles(n, seed=3, pid_base=1 << 40, start_in_generating_cell=False)
        ctx.locate()
        ctx.initial_setup()
        located = state(ctx)
        ctx.seed_particles(n, seed=3, pid_base=1 << 40, start_in_generating_cell=False)
        ctx.step()
        stepped = state(ctx)
        ctx.set_swarm(held)
        ctx.locate()
        ctx.initial_setup()
        same(located, state(ctx), "located first")
        ctx.set_swarm(held)
        ctx.step()
        same(stepped, state(ctx), "stepped at once")
