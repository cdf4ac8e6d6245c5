"""GPU: the interpolation of the same particles in a context of few slots, whose products stay on the FP64 pipe, and
of one slot more, whose products are the integer pipe's: the same bits, and the oracle's."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import PicContext, SwarmArrays
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FEW = 3 << 14


@pytest.mark.parametrize("n", [1, 63, 65, 5000, FEW])
def test_velocities_on_both_sides_of_the_line(require_gpu, n):
    IM, JM, KM = 9, 8, 15
    coor = W.bent_pipe_grid(IM, JM, KM)
    rng = np.random.default_rng(n)
    ucat = rng.standard_normal((KM, JM, IM, 3)) * 10.0 ** rng.integers(-12, 12, (KM, JM, IM, 3))
    ucat[2:4] *= 1e-300
    ucat[5, 3] = 0.0
    ucat[6, 2, 4] = [np.inf, -0.0, 5e-324]
    ucat[8, 5, 5] = [np.nan, 1e308, -1e308]
    pos, cell = W.volumetric_particles(coor, n, seed=n)
    w = rng.random((n, 3))
    special = rng.random((n, 3)) < 0.1
    w[special] = rng.choice([0.0, -0.0, 1.0, 1e-310, 2.0 ** -60, 1.0 - 2.0 ** -53, 2.0, -1.0, np.nan, np.inf], int(special.sum()))
    got = []
    for cap in (FEW, FEW + 1):
        with PicContext(0) as ctx:
            ctx.set_grid(coor)
            ctx.set_ucat(ucat)
            ctx.set_dt(0.0)
            ctx.reserve(cap)
            s = SwarmArrays.create(pos, cell=cell, status=1)
            s.weight[:] = w
            ctx.set_swarm(s)
            ctx.interpolate()
            held = ctx.get_swarm().sorted_by_pid()
            ctx.initial_setup()
            got.append((held.velocity, ctx.get_swarm().sorted_by_pid().velocity))
    for a, b in zip(*got):
        assert np.array_equal(a.view(np.int64), b.view(np.int64))
    g = O.Grid(coor)
    sw = O.Swarm.create(pos, cell=cell)
    sw.weight[:n] = w
    sw.status[:n] = 1
    O.interpolate(g, O.center_to_corner(g, W.node_sized(ucat)), sw)
    want = sw.view()["vel"]
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got[0][0]), nan)
    assert np.array_equal(got[0][0].view(np.int64)[~nan], want.view(np.int64)[~nan])
