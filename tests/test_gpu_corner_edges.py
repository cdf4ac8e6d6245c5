"""GPU: the plain corner field against the oracle, bit for bit, where a node has one, two, four or eight cells
in any direction, with components whose sums cancel, round, overflow, vanish or carry a sign of zero; and
the nodes a sparse swarm needs."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import PicContext, SwarmArrays
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 5, 3), (33, 2, 1), (31, 4, 9), (64, 3, 5)])
def test_corner_field_matches_the_oracle(require_gpu, dims):
    IM, JM, KM = dims
    coor = W.sinusoidal_grid(IM, JM, KM)
    rng = np.random.default_rng(IM)
    ucat = rng.standard_normal((KM, JM, IM, 3)) * 10.0 ** rng.integers(-20, 20, (KM, JM, IM, 3))
    near = rng.random((KM, JM, IM)) < 0.5          # values that cancel to a few units
    ucat[near] = np.where(rng.random((int(near.sum()), 3)) < 0.5, 1.0, -1.0) * (1.0 + 2.0 ** -52 * rng.integers(0, 4, (int(near.sum()), 3)))
    special = np.array([0.0, -0.0, 5e-324, -5e-324, 2.0 ** -1022, 2.0 ** -960, 1.7e308, -1.7e308, np.inf, np.nan])
    odd = rng.random((KM, JM, IM, 3)) < 0.05
    ucat[odd] = rng.choice(special, int(odd.sum()))
    ucat[..., 2] = np.where(rng.random((KM, JM, IM)) < 0.5, 0.0, -0.0) if JM == 4 else ucat[..., 2]
    g = O.Grid(coor)
    want = np.asarray(O.center_to_corner(g, W.node_sized(ucat))).reshape(KM + 1, JM + 1, IM + 1, 3)
    with PicContext(0) as ctx:
        ctx.set_grid(coor)
        ctx.set_ucat(ucat)
        got = ctx.get_corner()
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got.view(np.int64)[~nan], want.view(np.int64)[~nan])
        # one particle: the nodes of its cell alone are made, and its velocity is the oracle's
        for cell in {(0, 0, 0), (IM - 1, JM - 1, KM - 1), (IM // 2, 0, KM - 1)}:
            cent = W.cell_centroids(coor)[cell[2], cell[1], cell[0]]
            ctx.set_swarm(SwarmArrays.create(cent[None], cell=np.array([cell])))
            ctx.initial_setup()
            os_ = O.Swarm.create(cent[None], cell=np.array([cell]))
            sim = O.Simulation(g, W.node_sized(ucat), os_, 1e-3)
            sim.initial_setup()
            a, b = ctx.get_swarm().velocity, os_.view()["vel"]
            assert np.array_equal(np.isnan(a), np.isnan(b))
            assert np.array_equal(a.view(np.int64)[~np.isnan(a)], b.view(np.int64)[~np.isnan(b)]), cell
