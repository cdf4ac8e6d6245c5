"""GPU: the FP32 form's corner field and deposits on grids of every height around the columns its kernel carries
(four nodes), one cell thick included, against the plain form's."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import FORM_FP32, FORM_PLAIN_FP64, PicContext, SwarmArrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 3, 2), (5, 4, 3), (5, 4, 4), (5, 1, 5), (16, 15, 6), (17, 15, 7), (5, 4, 8)])
@pytest.mark.parametrize("per_cell", [0.5, 20])
def test_velocity_and_deposits_follow_the_plain_form(require_gpu, dims, per_cell):
    IM, JM, KM = dims
    coor = W.uniform_grid(IM, JM, KM)
    rng = np.random.default_rng(IM + JM + KM)
    ucat = rng.uniform(-1.0, 1.0, (KM, JM, IM, 3))
    n = int(per_cell * IM * JM * KM) + 1
    pos, cell = W.volumetric_particles(coor, n, seed=3)
    got = {}
    for form in (FORM_PLAIN_FP64, FORM_FP32):
        with PicContext(0) as ctx:
            ctx.set_form(form)
            ctx.set_grid(coor)
            ctx.set_ucat(ucat)
            ctx.set_dt(1e-3)
            ctx.set_swarm(SwarmArrays.create(pos, cell=cell))
            ctx.initial_setup()
            got[form] = (ctx.get_swarm().sorted_by_pid(), ctx.get_faces(), ctx.get_scattered())
    (a, fa, ca), (b, fb, cb) = got[FORM_PLAIN_FP64], got[FORM_FP32]
    assert np.array_equal(a.cell, b.cell) and np.array_equal(ca[0], cb[0])
    # FP32 roundings of the weights (1e-5 at most next to a face), of eight products and of the mean
    assert np.abs(a.velocity - b.velocity).max() <= 5e-5
    for x, y in zip(fa, fb):
        assert np.abs(x - y).max() <= 1e-5 * max(1.0, per_cell)
