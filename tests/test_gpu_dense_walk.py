"""GPU: steps of the FP32 and the learned form in contexts of as many slots as cells and of one more, whose
walks are compiled for more resident threads: the same results, bit for bit."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import FORM_FP32, FORM_LEARNED_FP32, PicContext, SwarmArrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [FORM_FP32, FORM_LEARNED_FP32])
@pytest.mark.parametrize("cfl", [0.5, 4.0])
def test_same_steps_on_both_sides_of_the_line(require_gpu, form, cfl):
    wl = W.config_bent_pipe(IM=12, JM=10, KM=48, n=5700, cfl=cfl, steps=1)
    cells = 12 * 10 * 48
    states = []
    for cap in (cells, cells + 1):
        with PicContext(0) as ctx:
            ctx.set_form(form)
            ctx.set_grid(wl.coor)
            ctx.set_ucat(wl.ucat)
            ctx.set_dt(wl.dt)
            ctx.reserve(cap)
            if form == FORM_LEARNED_FP32:
                ctx.locator_init(3)
                ctx.locator_min_distance(1.0)
            ctx.set_swarm(SwarmArrays.create(wl.pos, cell=wl.cell0))
            ctx.initial_setup()
            infos = [ctx.step() for _ in range(6)]
            s = ctx.get_swarm()
            states.append(([(i.n_end, i.removed_lost, i.removed_oob, i.walk_evals) for i in infos],
                           [s.position, s.velocity, s.weight, s.cell, s.pid, *ctx.get_faces()]))
    assert states[0][0] == states[1][0]
    for a, b in zip(states[0][1], states[1][1]):
        assert np.array_equal(a.view(np.int64), b.view(np.int64))
