"""GPU: vector fields between the callers' layout and the device's, at sizes around a thread block."""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from fdf_gb300.context import PicContext

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 2, 5), (8, 8, 4), (7, 5, 29), (16, 16, 33)])
@pytest.mark.parametrize("node_in", [False, True])
@pytest.mark.parametrize("node_out", [False, True])
def test_ucat_round_trip(require_gpu, dims, node_in, node_out):
    """Every bit comes back, whichever layout it went in by; the node layout's extra entries are zero."""
    IM, JM, KM = dims
    rng = np.random.default_rng(IM + 10 * JM + 100 * KM)
    u = rng.standard_normal((KM, JM, IM, 3)) * 10.0 ** rng.integers(-320, 300, (KM, JM, IM, 3))
    u.reshape(-1)[:3] = [-0.0, np.inf, -np.inf]
    full = rng.standard_normal((KM + 1, JM + 1, IM + 1, 3))
    full[:KM, :JM, :IM] = u
    with PicContext(0) as ctx:
        ctx.set_grid(W.uniform_grid(IM, JM, KM))
        ctx.set_ucat(full if node_in else u)
        got = ctx.get_ucat(node_sized=node_out)
    want = u
    if node_out:
        want = np.zeros((KM + 1, JM + 1, IM + 1, 3))
        want[:KM, :JM, :IM] = u
    assert np.array_equal(got.view(np.int64), want.view(np.int64))
