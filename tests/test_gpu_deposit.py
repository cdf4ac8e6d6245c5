"""GPU: the plain form's deposits against the oracle, bit for bit, from empty to crowded cells: the sums staged in
shared memory and not, warps that mix both, rows that end inside a warp."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import PicContext, SwarmArrays
from oracle import oracle as O
from tests.parity_util import assert_faces_bitwise, from_oracle_swarm, to_oracle_swarm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("momentum", [False, True])
@pytest.mark.parametrize("dims", [(33, 5, 7), (16, 12, 9)])
@pytest.mark.parametrize("per_cell", [0.02, 0.3, 1.2, 4.4, 5.5, 30.0])
def test_deposits_match_the_oracle(require_gpu, momentum, dims, per_cell):
    IM, JM, KM = dims
    coor = W.bent_pipe_grid(IM, JM, KM)
    n = max(int(per_cell * IM * JM * KM), 1)
    pos, cell = W.volumetric_particles(coor, n, seed=int(10 * per_cell) + IM)
    rng = np.random.default_rng(n)
    # a third of the particles in one corner of the grid: cells far above the mean next to empty ones
    crowd = rng.random(n) < 0.33
    far = ~crowd & (cell[:, 0] < IM // 3)
    pos, cell = pos[~far], cell[~far]
    n = len(pos)
    cent = W.cell_centroids(coor)
    ucat = W.field_pipe(coor, cent)
    ucat[..., 2] = 0.0   # a component that is zero everywhere
    with PicContext(0) as ctx:
        ctx.set_grid(coor)
        ctx.set_ucat(ucat)
        ctx.set_dt(1e-3)
        ctx.set_volume(0.37)
        if momentum:
            ctx.set_momentum_deposit(True)
        P = 101325.0 * rng.uniform(0.5, 1.5, n)
        ctx.set_swarm(SwarmArrays.create(pos, cell=cell, P=P, pid=rng.permutation(n)))
        s0 = ctx.get_swarm()
        ctx.initial_setup()
        g, os_ = O.Grid(coor), to_oracle_swarm(s0)
        sim = O.Simulation(g, W.node_sized(ucat), os_, 1e-3)
        sim.initial_setup()
        ref = O.deposit_faces(g, os_, volume=0.37, momentum=momentum)
        assert_faces_bitwise(ctx.get_faces(), ref, what="faces")
        if momentum:
            for gm, key in zip(ctx.get_face_momentum(), ("mom_i", "mom_j", "mom_k")):
                assert np.array_equal(gm.view(np.int64), ref[key].view(np.int64)), key
        # the P average sums each cell's particles by PID, as the faces do (the oracle's scatter takes the
        # swarm's own order, which is another here)
        s = from_oracle_swarm(os_).sorted_by_pid()
        c = (s.cell[:, 2] * (JM + 1) + s.cell[:, 1]) * (IM + 1) + s.cell[:, 0]
        total = np.zeros(sim.avg.size)
        np.add.at(total, c, s.P)
        num = np.bincount(c, minlength=total.size)
        want = np.where(num > 0, total / np.maximum(num, 1), 0.0).reshape(sim.avg.shape)
        count, avg = ctx.get_scattered()
        assert np.array_equal(count, sim.count) and np.array_equal(avg, want)
