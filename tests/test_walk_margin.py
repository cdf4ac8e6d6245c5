"""CPU: the walk's one margin per cell (fdf_walk.cuh), restated in numpy.

An evaluation whose six FP32 distances all exceed the cell's margin M takes their signs as the
classes; the others go through the faces' own margins M_f and the exact FP64 distance.  That is
the M_f rule's outcome exactly when no face with |d32| <= M_f has |d32| > M, which is checked here
for points around the cells of curved grids, next to a cell's first vertex, within a few ulps of a
face plane, and far from the origin (where the positions' roundings carry the margins).
"""
import numpy as np
import pytest

from fdf_gb300 import workloads as W
from tests.test_walk_bound import F, OFF, U, f32, fma32, kernel_d32, planes_of, rows_of


def cell_margin(p, v, thr, sigma):
    """M for positions p [n][3], as k_build_table32 and walk_ref32 compute it."""
    c0h = f32(v[:, 0])
    size = np.sum(np.abs(c0h.astype(np.float64)), axis=1)
    slack = sigma * 2.0 ** -48 + size * 40.0 * 2.0 ** -48
    base = np.nextafter(f32((thr + slack) * (1.0 + 2.0 ** -19)), F(np.inf))
    ph = f32(p)
    pl = f32(p - ph.astype(np.float64))
    c0l = f32(v[:, 0] - c0h.astype(np.float64))
    pr = np.abs(f32(f32(ph - c0h) + f32(pl - c0l)))
    a = np.abs(ph)
    X = f32(f32(f32(a[:, 0] + a[:, 1]) + a[:, 2]) * F(40.0 * U * U))
    s = f32(f32(pr[:, 0] + pr[:, 1]) + pr[:, 2])
    return fma32(s, np.full_like(s, F(40.0 * U)), f32(base + X))


@pytest.mark.parametrize("grid,shift", [("sinusoidal", 0.0), ("bent_pipe", 0.0), ("bent_pipe", 1.0e4)])
def test_cell_margin_covers_face_margins(grid, shift):
    coor = (W.sinusoidal_grid(24, 20, 64, amp=0.08) if grid == "sinusoidal" else W.bent_pipe_grid(16, 16, 96)) + shift
    KM, JM, IM = (s - 1 for s in coor.shape[:3])
    rng = np.random.default_rng(5)
    m = 4000
    ijk = np.stack([rng.integers(0, IM, m), rng.integers(0, JM, m), rng.integers(0, KM, m)], 1)
    v = np.stack([coor[ijk[:, 2] + o[2], ijk[:, 1] + o[1], ijk[:, 0] + o[0]] for o in OFF], 1)
    fc, n = planes_of(v)
    h = np.linalg.norm(v[:, 6] - v[:, 0], axis=1)
    thr = 1e-11 * h
    c0h, c0l, thr32, slack, n32, e32, sigma = rows_of(v, fc, n, thr)
    settled = total = 0
    for trial in range(9):
        lo, hi = v.min(1), v.max(1)
        if trial < 3:
            p = lo + rng.uniform(-1.0, 2.0, lo.shape) * (hi - lo)
        elif trial < 5:
            p = v[:, 0] + rng.standard_normal((m, 3)) * (1e-9 * h)[:, None]
        else:   # within a few units of the margins of a face plane, on either side
            f = rng.integers(0, 6, m)
            nf, fcf = n[np.arange(m), f], fc[np.arange(m), f]
            t = rng.standard_normal((m, 3))
            t -= np.einsum("ij,ij->i", t, nf)[:, None] * nf
            off = rng.uniform(-60.0, 60.0, m) * U * (h + U * np.abs(fcf).sum(1))
            p = fcf + 0.3 * h[:, None] * t + off[:, None] * nf
        d32, S, Mf, _ = kernel_d32(p, c0h, c0l, thr32, slack, n32, e32)
        M = cell_margin(p, v, thr, sigma)[:, None]
        open_f = ~(np.abs(d32) > Mf)
        assert not np.any(open_f & (np.abs(d32) > M))
        settled += int(np.all(np.abs(d32) > M, axis=1).sum())
        total += m
    assert settled / total > 0.2   # the near-plane and near-vertex points are meant to stay open
