"""GPU: the plain form's deposits on both sides of the sizes that give a node's four chains blocks of their own (the
nodes, with the capacity against five times the cells), against the oracle bit for bit, cells crowded and
empty."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import PicContext, SwarmArrays
from oracle import oracle as O
from tests.parity_util import assert_faces_bitwise, to_oracle_swarm

pytestmark = pytest.mark.gpu


# 32768 and 33792 nodes; 524,880 nodes (above half a million) and 518,400
@pytest.mark.parametrize("dims,per_cell,room", [((31, 31, 31), 0.4, 1), ((31, 31, 32), 0.4, 1), ((31, 31, 31), 7.0, 1),
                                                ((31, 31, 32), 7.0, 1), ((31, 31, 32), 0.4, 20), ((1, 1, 3), 900.0, 1),
                                                ((80, 79, 79), 0.2, 30), ((80, 79, 80), 0.2, 30)])
@pytest.mark.parametrize("momentum", [False, True])
def test_deposits_on_both_sides(require_gpu, dims, per_cell, room, momentum):
    IM, JM, KM = dims
    coor = W.sinusoidal_grid(IM, JM, KM, amp=0.02)
    n = int(per_cell * IM * JM * KM)
    pos, cell = W.volumetric_particles(coor, n, seed=IM + KM)
    rng = np.random.default_rng(n)
    stay = (cell[:, 0] >= IM // 3) | (rng.random(n) < 0.5)   # a thin part and a full one
    crowd = np.repeat(np.flatnonzero(stay)[:7], 150)          # and a few cells far above the others
    pos, cell = np.concatenate([pos[stay], pos[crowd]]), np.concatenate([cell[stay], cell[crowd]])
    n = len(pos)
    ucat = W.field_taylor_green(W.cell_centroids(coor))
    P = 101325.0 * rng.uniform(-0.5, 1.5, n)
    with PicContext(0) as ctx:
        ctx.set_grid(coor)
        ctx.set_ucat(ucat)
        ctx.set_dt(1e-3)
        ctx.set_volume(0.37)
        ctx.set_momentum_deposit(momentum)
        ctx.reserve(room * n)
        ctx.set_swarm(SwarmArrays.create(pos, cell=cell, P=P, pid=rng.permutation(n)))
        ctx.initial_setup()
        s = ctx.get_swarm()   # sorted by (cell, PID): the order of every sum
        ref = O.deposit_faces(O.Grid(coor), to_oracle_swarm(s), volume=0.37, momentum=momentum)
        assert_faces_bitwise(ctx.get_faces(), ref, what="faces")
        if momentum:
            for gm, key in zip(ctx.get_face_momentum(), ("mom_i", "mom_j", "mom_k")):
                assert np.array_equal(gm.view(np.int64), ref[key].view(np.int64)), key
        in_cell = s.cell[:, 0] >= 0
        c = ((s.cell[:, 2] * (JM + 1) + s.cell[:, 1]) * (IM + 1) + s.cell[:, 0])[in_cell]
        nodes = (KM + 1) * (JM + 1) * (IM + 1)
        total, num = np.zeros(nodes), np.bincount(c, minlength=nodes)
        np.add.at(total, c, s.P[in_cell])
        count, avg = ctx.get_scattered()
        assert np.array_equal(count.ravel(), num)
        assert np.array_equal(avg.ravel(), np.where(num > 0, total / np.maximum(num, 1), 0.0))
