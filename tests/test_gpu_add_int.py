"""GPU: a + b on the integer pipe (fdf_exact.cuh) against the hardware, bit for bit, at the operands its bit
arithmetic turns on: every distance of exponents, significands of every length with zero, all-ones and
single-bit tails (ties, carries), near and full cancellation, and what is handed on."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from fdf_gb300 import build as B

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory, require_gpu):
    out = str(tmp_path_factory.mktemp("add_int") / "libadd_int_selftest.so")
    src = os.path.join(HERE, "kernels", "add_int_selftest.cu")
    r = subprocess.run([B.nvcc()] + B.NVFLAGS + ["-I", B.CSRC, "-shared", src, "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(out)


def significands(rng, n):
    """1 to 53 leading bits, then zeros, ones or one bit."""
    keep = rng.integers(0, 53, n).astype(np.uint64)
    low = (np.uint64(1) << (np.uint64(52) - keep)) - np.uint64(1)
    f = rng.integers(0, 1 << 52, n, dtype=np.uint64) & ~low
    tail = np.where(rng.integers(0, 2, n) == 1, low, np.uint64(1)) * rng.integers(0, 2, n, dtype=np.uint64)
    return f | (tail & low)


def doubles(rng, e):
    n = e.size
    sign = rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63)
    return (sign | (e.astype(np.uint64) << np.uint64(52)) | significands(rng, n)).view(np.float64)


@pytest.mark.parametrize("what", ["distances", "cancellation", "range", "special"])
def test_integer_addition_at_its_edges(lib, what):
    rng = np.random.default_rng(12)
    n = 2_000_000
    if what == "distances":      # every exponent distance up to past the significand, both ways, both signs
        e = rng.integers(200, 1800, n)
        a, b = doubles(rng, e), doubles(rng, e + rng.integers(-70, 71, n))
    elif what == "cancellation":   # a and -a a few units, or a few exponents, apart
        a = doubles(rng, rng.integers(60, 2046, n))
        u = a.view(np.uint64) ^ np.uint64(1 << 63)
        b = (u + (np.uint64(1) << rng.integers(0, 54, n, dtype=np.uint64)) * rng.integers(0, 3, n, dtype=np.uint64)
             - rng.integers(0, 3, n, dtype=np.uint64)).view(np.float64)
    elif what == "range":        # both ends of the exponents
        e = np.where(rng.integers(0, 2, n) == 1, rng.integers(0, 130, n), rng.integers(1980, 2048, n))
        a, b = doubles(rng, e), doubles(rng, np.clip(e + rng.integers(-66, 67, n), 0, 2047))
    else:
        v = np.array([0.0, 1.0, np.nextafter(1.0, 0.0), np.nextafter(1.0, 2.0), 2.0 ** -53, 1.5 * 2.0 ** -53, 2.0 ** -54,
                      np.nextafter(2.0 ** -53, 1.0), np.nextafter(2.0 ** -54, 1.0), 2.0 ** -959, 2.0 ** -958, 2.0 ** -1022,
                      5e-324, np.inf, np.nan, np.finfo(np.float64).max, 2.0 ** 1023, 2.0 ** 1022, 2.0 ** 970, 2.0 ** 969])
        v = np.concatenate([v, -v])
        a, b = np.repeat(v, v.size), np.tile(v, v.size)
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    bad = np.zeros(1, dtype=np.uint64)
    p = lambda x: ctypes.c_void_p(x.ctypes.data)  # noqa: E731
    assert lib.fdf_test_add_int(p(a), p(b), ctypes.c_longlong(a.size), p(bad)) == 0
    assert bad[0] == 0, f"{bad[0]} of {a.size} sums differ"
