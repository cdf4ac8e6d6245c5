"""GPU: 1 - a and a * b on the integer pipe (fdf_exact.cuh) against the hardware, bit for bit, at the operands
their bit arithmetic turns on: every exponent of (0, 1], significands of every length with all-ones and
single-bit tails (ties and carries), the first and last values of each range, and what is handed on."""
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
    out = str(tmp_path_factory.mktemp("one_minus") / "libone_minus_selftest.so")
    src = os.path.join(HERE, "kernels", "one_minus_selftest.cu")
    r = subprocess.run([B.nvcc()] + B.NVFLAGS + ["-I", B.CSRC, "-shared", src, "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(out)


@pytest.mark.parametrize("what", ["exponents", "significands", "special"])
def test_integer_pipe_arithmetic_at_its_edges(lib, what):
    rng = np.random.default_rng(11)
    if what == "exponents":      # every exponent up to 1, and a few above
        e = np.repeat(np.arange(0, 1030, dtype=np.uint64), 512)
        a = ((e << np.uint64(52)) | rng.integers(0, 1 << 52, e.size, dtype=np.uint64)).view(np.float64)
    elif what == "significands":   # 1 to 53 leading bits, then zeros, ones, or one bit
        e = rng.integers(940, 1023, 400_000).astype(np.uint64)
        keep = rng.integers(0, 53, e.size).astype(np.uint64)
        low = (np.uint64(1) << (np.uint64(52) - keep)) - np.uint64(1)
        f = rng.integers(0, 1 << 52, e.size, dtype=np.uint64) & ~low
        tail = np.where(rng.integers(0, 2, e.size) == 1, low, np.uint64(1)) * rng.integers(0, 2, e.size, dtype=np.uint64)
        a = ((e << np.uint64(52)) | (f | (tail & low))).view(np.float64)
    else:
        v = [0.0, -0.0, 1.0, np.nextafter(1.0, 0.0), np.nextafter(1.0, 2.0), 2.0, -1.0, 0.5, 2.0 ** -53, 2.0 ** -54, 2.0 ** -55,
             1.5 * 2.0 ** -54, 3 * 2.0 ** -55, 2.0 ** -1022, 5e-324, np.inf, -np.inf, np.nan, 1e300, 1e-300, 2.0 ** -11,
             np.nextafter(2.0 ** -11, 0.0), np.nextafter(2.0 ** -11, 1.0)]
        a = np.repeat(np.array(v), len(v))
    b = np.tile(np.array(v), len(v)) if what == "special" else rng.permutation(a)
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    bad = np.zeros(2, dtype=np.uint64)
    p = lambda x: ctypes.c_void_p(x.ctypes.data)  # noqa: E731
    assert lib.fdf_test_one_minus(p(a), p(b), ctypes.c_longlong(a.size), p(bad)) == 0
    assert bad[0] == 0, f"{bad[0]} differences from 1.0 - a"
    assert bad[1] == 0, f"{bad[1]} products differ"
