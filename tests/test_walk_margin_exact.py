"""CPU: the walk's one margin per cell with the row's base rounded up exactly as the kernel rounds it
(__double2float_ru): the next float only where the nearest one is below the value.  A base one unit too large makes
the margin larger, and what is checked of it (no open face above the margin) easier."""
import numpy as np
import pytest

import tests.test_walk_margin as T
from tests.test_walk_bound import F, U, f32, fma32


def round_up(v):
    near = f32(v)
    return np.where(near.astype(np.float64) < v, np.nextafter(near, F(np.inf)), near).astype(F)


def cell_margin(p, v, thr, sigma):
    """M for positions p [n][3], as k_build_table32 and walk_ref32 compute it."""
    c0h = f32(v[:, 0])
    size = np.sum(np.abs(c0h.astype(np.float64)), axis=1)
    slack = sigma * 2.0 ** -48 + size * (40.0 * 2.0 ** -48)
    base = round_up((thr + slack) * (1.0 + 2.0 ** -19))
    ph = f32(p)
    pl = f32(p - ph.astype(np.float64))
    c0l = f32(v[:, 0] - c0h.astype(np.float64))
    pr = np.abs(f32(f32(ph - c0h) + f32(pl - c0l)))
    a = np.abs(ph)
    X = f32(f32(f32(a[:, 0] + a[:, 1]) + a[:, 2]) * F(40.0 * U * U))
    s = f32(f32(pr[:, 0] + pr[:, 1]) + pr[:, 2])
    return fma32(s, np.full_like(s, F(40.0 * U)), f32(base + X))


def test_round_up():
    v = np.array([1.0, 1.0 + 2.0 ** -30, 1.0 + 2.0 ** -23, 1.0 + 1.5 * 2.0 ** -23 - 2.0 ** -40, 3e-11, 0.0])
    up = round_up(v).astype(np.float64)
    assert np.all(up >= v) and np.all(np.nextafter(round_up(v), F(-np.inf)).astype(np.float64) < v)
    assert up[0] == 1.0 and up[2] == v[2]


@pytest.mark.parametrize("grid,shift", [("sinusoidal", 0.0), ("bent_pipe", 0.0), ("bent_pipe", 1.0e4)])
def test_cell_margin_covers_face_margins(monkeypatch, grid, shift):
    loose, smaller = T.cell_margin, []

    def exact(p, v, thr, sigma):
        m = cell_margin(p, v, thr, sigma)
        smaller.append(np.any(m < loose(p, v, thr, sigma)))
        assert np.all(m <= loose(p, v, thr, sigma))
        return m

    monkeypatch.setattr(T, "cell_margin", exact)
    T.test_cell_margin_covers_face_margins(grid, shift)
    assert any(smaller) or shift   # far from the origin the positions' part hides the base's last unit
