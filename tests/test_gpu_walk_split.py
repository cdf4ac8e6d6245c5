"""GPU: the plain walk's weights on both sides of the slot count from which two products of each distance
go to the integer pipe, against the walk of the same points outside the swarm (no such products) and the
oracle."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import PicContext, SwarmArrays
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LINE = 3 << 19


@pytest.mark.parametrize("n", [LINE - 1, LINE, LINE + 129])
def test_weights_are_the_same_on_both_sides_of_the_line(require_gpu, n):
    IM, JM, KM = 21, 13, 40
    coor = W.bent_pipe_grid(IM, JM, KM) * 1e3   # products of all exponents up to the pipe's length
    pos, cell = W.volumetric_particles(coor, n, seed=5)
    rng = np.random.default_rng(n)
    start = np.clip(cell + rng.integers(-2, 3, cell.shape), 0, [IM - 1, JM - 1, KM - 1])
    pos[:6] = [[0.0, 0.0, 0.0], [1e-310, 0.0, -1e-310], [1e300, 1.0, 1.0], [np.inf, 0.0, 0.0], [np.nan, 1.0, 2.0], coor[3, 3, 3]]
    with PicContext(0) as ctx:
        ctx.set_grid(coor)
        ctx.set_ucat(np.zeros((KM, JM, IM, 3)))
        ctx.set_swarm(SwarmArrays.create(pos, cell=start, status=0))
        ctx.locate()
        s = ctx.get_swarm()
        got, w, st = ctx.locate_points(pos, start)
    order = np.argsort(s.pid)
    assert np.array_equal(s.cell[order], got)
    assert np.array_equal(s.status[order], st)
    at = st == 1
    assert at.sum() > 0.9 * n
    assert np.array_equal(s.weight[order][at].view(np.int64), w[at].view(np.int64))
    g = O.Grid(coor)
    for p in rng.integers(6, n, 60):
        r = O.locate_particle(g, pos[p], start[p])
        assert np.array_equal(got[p], r["cell"]) and st[p] == r["status"], p
        if st[p] == 1:
            assert np.array_equal(w[p].view(np.int64), r["weights"].view(np.int64)), p
