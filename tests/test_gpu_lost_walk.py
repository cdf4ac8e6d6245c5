"""GPU: the FP32 form's step for particles without a cell, whose walks from cell (0,0,0) evaluate the cells
that the margins leave open inside the loop, against the same particles with (0,0,0) as their previous cell,
whose walks do so after it."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import FORM_FP32, PicContext, SwarmArrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n", [((6, 5, 400), 20_000), ((40, 30, 7), 20_000), ((3, 3, 3), 33)])
def test_particles_without_a_cell_walk_from_the_first(require_gpu, dims, n):
    IM, JM, KM = dims
    coor = W.sinusoidal_grid(IM, JM, KM)
    pos, _ = W.volumetric_particles(coor, n, seed=8)
    rng = np.random.default_rng(n)
    nodes = coor.reshape(-1, 3)
    on = rng.random(n) < 0.2          # on the nodes: within every margin of their walks' last faces
    pos[on] = nodes[rng.integers(0, len(nodes), int(on.sum()))]
    pos[:3] = [[1e6, 0.0, 0.0], [np.nan, 0.0, 0.0], [0.0, np.inf, 0.0]]
    none = rng.random(n) < 0.5        # warps that mix both
    states = []
    for lost in (np.zeros(n, bool), none, np.ones(n, bool)):
        cell = np.zeros((n, 3), np.int64)
        cell[lost] = -1
        with PicContext(0) as ctx:
            ctx.set_form(FORM_FP32)
            ctx.set_grid(coor)
            ctx.set_ucat(np.zeros((KM, JM, IM, 3)))
            ctx.set_dt(0.0)
            ctx.set_swarm(SwarmArrays.create(pos, cell=cell, status=0))
            info = ctx.step()
            s = ctx.get_swarm().sorted_by_pid()
            states.append((s, info))
    a, ia = states[0]
    assert a.n > 0 and ia.removed_lost > 0
    for b, ib in states[1:]:
        assert (ia.walk_evals, ia.removed_lost, ia.removed_oob, ia.n_end) == (ib.walk_evals, ib.removed_lost, ib.removed_oob, ib.n_end)
        assert np.array_equal(a.pid, b.pid) and np.array_equal(a.cell, b.cell) and np.array_equal(a.status, b.status)
        for x, y in ((a.position, b.position), (a.weight, b.weight)):
            assert np.array_equal(x.view(np.int64), y.view(np.int64))
