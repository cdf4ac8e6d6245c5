"""GPU: caller-held points at the sizes where the calls change route: one point, a block's edge, and the
number from which the interpolation makes the whole corner field instead of each point's corners; and
calls of growing and shrinking size on one context."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import PicContext
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_points_at_the_edges_of_the_routes(require_gpu):
    IM, JM, KM = 9, 7, 11
    coor = W.sinusoidal_grid(IM, JM, KM)
    rng = np.random.default_rng(2)
    ucat = rng.standard_normal((KM, JM, IM, 3))
    ucat[0, 0, 0] = [0.0, -0.0, 1e-310]
    nodes = (IM + 1) * (JM + 1) * (KM + 1)
    g = O.Grid(coor)
    corner = O.center_to_corner(g, W.node_sized(ucat))
    with PicContext(0) as ctx:
        ctx.set_grid(coor)
        ctx.set_ucat(ucat)
        for n in (1, 127, 128, 129, nodes // 8 - 1, nodes // 8, nodes // 8 + 1, 3000, 5, 3001):
            pos, cell = W.volumetric_particles(coor, n, seed=n)
            start = np.clip(cell + rng.integers(-2, 3, cell.shape), -1, [IM, JM, KM])   # some outside: from (0,0,0)
            got, w, st = ctx.locate_points(pos, start)
            vel = ctx.interpolate_points(got, w)
            sw = O.Swarm.create(pos, cell=got)
            sw.weight[:n] = w
            sw.status[:n] = st
            O.interpolate(g, corner, sw)
            assert np.array_equal(vel.view(np.int64), sw.view()["vel"].view(np.int64)), n
            for p in rng.integers(0, n, 40):
                inside = np.all((start[p] >= 0) & (start[p] < [IM, JM, KM]))
                r = O.locate_particle(g, pos[p], start[p] if inside else (-1, -1, -1))
                assert np.array_equal(got[p], r["cell"]) and st[p] == r["status"], (n, p)
                assert np.array_equal(w[p].view(np.int64), r["weights"].view(np.int64)), (n, p)
        # weights outside [0, 1] and not finite, cells outside the grid: as the corner field's route
        n = nodes // 8 + 1
        cell = rng.integers(-1, 12, (n, 3))
        w = rng.uniform(-0.5, 1.5, (n, 3))
        w[:6] = [[np.nan, 0.5, 0.5], [np.inf, 0.1, 0.2], [-np.inf, 1.0, 1.0], [0.0, -0.0, 1.0], [1e-320, 0.3, 0.4], [1.0, 1.0, 1.0]]
        many = ctx.interpolate_points(cell, w)
        few = np.concatenate([ctx.interpolate_points(cell[a:a + 50], w[a:a + 50]) for a in range(0, n, 50)])
        assert np.array_equal(many.view(np.int64), few.view(np.int64))
