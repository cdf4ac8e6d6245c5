"""Training: a step's two kernels begin before the ones ahead of them have ended and wait before they touch
what those write.

CPU: no pointer to such memory may be `__restrict__` (the compiler could move its loads past the wait or
take the read-only path); the samples, which no step writes, may.
GPU: several hundred steps are bit for bit the same steps made one call at a time, every kernel after the
end of the one before: gradients from fdf_LocatorGradients, Adam in FP32 on the host.
"""
import math
import os
import re

import numpy as np
import pytest

from fdf_gb300 import workloads as W

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fdf_gb300", "csrc", "fdf_mlp.cu")


def test_no_restrict_on_what_the_kernel_ahead_writes():
    text = open(SRC).read()
    found = {}
    for m in re.finditer(r"__global__ void (?:__launch_bounds__\([^)]*\)\s*)?(\w+)\(([^{]*)\)\s*\{(.*?)\n\}\n", text, re.S):
        name, params, body = m.groups()
        if "await_previous()" in body:
            found[name] = [p.split("__restrict__")[1].strip() for p in params.split(",") if "__restrict__" in p]
    assert set(found) == {"k_train_tc", "k_train_update"}
    assert found["k_train_update"] == []
    assert set(found["k_train_tc"]) <= {"xs", "ts"}


def _mix64(z):
    with np.errstate(over="ignore"):
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def _batch(seed, step, B, n):
    with np.errstate(over="ignore"):
        base = _mix64(np.uint64(seed ^ 0x5DEECE66D) * np.uint64(0xD1B54A32D192ED03) + np.uint64(step))
        return (_mix64(base + np.arange(B, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)) % np.uint64(n)).astype(np.int64)


@pytest.mark.gpu
@pytest.mark.parametrize("B,steps", [(16, 300), (400, 300), (8192, 40)])
def test_steps_as_one_call_at_a_time(require_gpu, B, steps):
    from fdf_gb300.context import PicContext
    f = np.float32
    coor = W.bent_pipe_grid(12, 12, 48)
    dims = np.array([12, 12, 48])
    n, seed, lr = 20_000, 9, 2e-3
    with PicContext(0) as ctx:
        ctx.set_grid(coor)
        ctx.locator_init(7)
        w = ctx.locator_get_params()
        hist = ctx.locator_train(n, seed=seed, steps=steps, batch=B, lr=lr)
        got = ctx.locator_get_params()
        pos, cell = W.volumetric_particles(coor, n, seed)
        at, _, status = ctx.locate_points(pos, cell)
        pos, at = pos[status == 1], at[status == 1]
        centre, inv_half = ctx.locator_normalization()
        xs = (pos.astype(f) - centre) * inv_half
        ts = f(2.0) * (at.astype(f) + f(0.5)) / dims.astype(f) - f(1.0)
        m, v = np.zeros_like(w), np.zeros_like(w)
        for t in range(steps):
            q = _batch(seed, t, B, len(pos))
            ctx.locator_set_params(w)
            g, loss = ctx.locator_gradients(xs[q], ts[q])
            assert f(loss) == hist[t], t
            m = f(0.9) * m + f(0.1) * g
            v = f(0.999) * v + f(0.001) * g * g
            c1, c2 = f(1.0 - math.pow(0.9, t + 1)), f(1.0 - math.pow(0.999, t + 1))
            lr_t = f(lr * (0.02 + 0.98 * 0.5 * (1.0 + math.cos(math.pi * t / steps))))
            w = w - lr_t * (m / c1) / (np.sqrt(v / c2) + f(1e-8))
            assert w.dtype == f
        assert np.array_equal(got, w)
