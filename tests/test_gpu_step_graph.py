"""GPU: single steps, which replay a captured step after the first few, through every change between them."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import FORM_FP32, FORM_PLAIN_FP64, PicContext, SwarmArrays
from oracle import oracle as O
from tests.parity_util import assert_swarm_bitwise, from_oracle_swarm, to_oracle_swarm

pytestmark = pytest.mark.gpu


def test_replayed_steps_follow_every_change(require_gpu):
    """Time step, velocity, swarm (fewer particles), volume and momentum deposit change between steps;
    after each change seven steps with their counts read match the oracle's, bit for bit."""
    wl = W.config_bent_pipe(IM=12, JM=10, KM=48, n=4000, cfl=0.5, steps=1)
    other = 0.5 * wl.ucat + 0.01
    with PicContext(0) as ctx:
        ctx.load_workload(wl)
        ctx.reserve(5000)
        ctx.set_swarm(SwarmArrays.create(wl.pos, cell=wl.cell0))
        g, os_ = O.Grid(wl.coor), to_oracle_swarm(ctx.get_swarm())
        sim = O.Simulation(g, wl.ucat_node_sized(), os_, wl.dt)
        ctx.initial_setup()
        sim.initial_setup()

        def seven(what):
            for q in range(7):
                i, o = ctx.step(), sim.step()
                assert (i.n_end, i.removed_lost, i.removed_oob, i.walk_evals) == (os_.n, o.removed_lost, o.removed_oob, o.evals)
                assert i.n_start == i.n_end + i.removed_lost + i.removed_oob
            assert_swarm_bitwise(ctx.get_swarm(), from_oracle_swarm(os_), what)

        seven("first")
        ctx.set_dt(0.5 * wl.dt)
        sim.dt = 0.5 * wl.dt
        seven("another time step")
        ctx.set_ucat(other)
        sim.ucat = W.node_sized(other)
        seven("another velocity")
        ctx.set_momentum_deposit(True)
        ctx.set_volume(2.0)
        seven("another deposit")
        ref = O.deposit_faces(g, os_, volume=2.0, momentum=True)
        assert np.array_equal(ctx.get_face_momentum()[0].view(np.int64), ref["mom_i"].view(np.int64))
        s = SwarmArrays.create(wl.pos[:1500], cell=wl.cell0[:1500])
        ctx.set_swarm(s)
        os_ = to_oracle_swarm(ctx.get_swarm())
        sim = O.Simulation(g, W.node_sized(other), os_, 0.5 * wl.dt)
        seven("another swarm, not located before its first step")


def test_form_changes_between_replayed_steps(require_gpu):
    """A swarm of another form after captured steps: as in a context of its own."""
    wl = W.config_bent_pipe(IM=12, JM=10, KM=48, n=4000, cfl=0.5, steps=1)
    outs = []
    for forms in ([FORM_FP32], [FORM_PLAIN_FP64, FORM_FP32], [FORM_FP32, FORM_PLAIN_FP64, FORM_FP32]):
        with PicContext(0) as ctx:
            ctx.load_workload(wl, form=forms[0])
            for form in forms:
                ctx.set_form(form)
                ctx.set_swarm(SwarmArrays.create(wl.pos, cell=wl.cell0))
                ctx.initial_setup()
                for _ in range(9):
                    ctx.step(info=False)
            outs.append((ctx.get_swarm(), ctx.get_faces()))
    for s, faces in outs[1:]:
        assert_swarm_bitwise(s, outs[0][0], "form change")
        assert all(np.array_equal(a, b) for a, b in zip(faces, outs[0][1]))
