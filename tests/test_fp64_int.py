"""The integer FP64 product and comparisons against the host's IEEE ones, bit
for bit: any patterns, ties and near ties, powers of two, results at the ends
of the range, zeros, infinities and NaN."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HARNESS = r"""
#include "fp64_int.cuh"
extern "C" void eval(const double* a, const double* b, double* q, double* u, unsigned char* c, long n) {
    for (long i = 0; i < n; ++i) {
        q[i] = tflows::mul_rn(a[i], b[i]);
        u[4 * i] = tflows::twice(a[i]);
        u[4 * i + 1] = tflows::half(a[i]);
        u[4 * i + 2] = tflows::zero_plus(a[i]);
        u[4 * i + 3] = tflows::signed_by(tflows::zero_minus(a[i]), true);
        c[i] = tflows::less(a[i], b[i]) | tflows::above_zero(a[i]) << 1 | tflows::below_zero(a[i]) << 2;
    }
}
"""


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    d = tmp_path_factory.mktemp("mul")
    (d / "h.cpp").write_text(HARNESS)
    so = d / "h.so"
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-x", "c++",
                    "-I", os.path.join(ROOT, "t-flows-old-compressible_gb300", "csrc"),
                    str(d / "h.cpp"), "-o", str(so)], check=True)
    fn = ctypes.CDLL(str(so)).eval
    p = ctypes.c_void_p

    def run(a, b):
        q, u, c = np.empty_like(a), np.empty((a.size, 4)), np.empty(a.size, np.uint8)
        fn(*(p(v.ctypes.data) for v in (a, b, q, u, c)), ctypes.c_long(a.size))
        return np.column_stack([q, u]), c
    return run


def _near(rng, n):
    """Significands of few bits or near a power of two, exponents of any kind."""
    one = np.uint64(1) << np.uint64(52)
    f = [rng.integers(0, 8, n, dtype=np.uint64), one - np.uint64(1) - rng.integers(0, 8, n, dtype=np.uint64),
         rng.integers(0, 2**27, n, dtype=np.uint64) << np.uint64(25),
         rng.integers(0, 2**26, n, dtype=np.uint64) << np.uint64(26), rng.integers(0, 2**52, n, dtype=np.uint64)]
    e = [rng.integers(0, 2048, n, dtype=np.uint64), rng.integers(1020, 1027, n, dtype=np.uint64),
         rng.integers(505, 520, n, dtype=np.uint64), rng.integers(1530, 1540, n, dtype=np.uint64)]
    out = [(a | b << np.uint64(52)) | rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63)
           for a in f for b in e]
    return rng.permutation(np.concatenate(out)).view(np.float64)


SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308,
                    1.7976931348623157e308, 1.0, -1.0, 0.5, 2.0, 1.5e-154, 1.3e154])


@pytest.mark.parametrize("kind", ["any", "near", "special"])
def test_products_and_comparisons(evaluate, kind):
    rng = np.random.default_rng(3)
    if kind == "any":
        a, b = (rng.integers(0, 2**64, 600_000, dtype=np.uint64).view(np.float64) for _ in range(2))
    elif kind == "near":
        a, b = _near(rng, 30_000), _near(rng, 30_000)
        b[::7] = a[::7]
        b[::11] = -a[::11]
    else:
        a, b = (np.ascontiguousarray(v.ravel()) for v in np.meshgrid(SPECIAL, SPECIAL))
    with np.errstate(all="ignore"):
        want = np.column_stack([a * b, 2.0 * a, 0.5 * a, 0.0 + a, -(0.0 - a)])
    got, c = evaluate(a, b)
    same = (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))
    bad = ~same.all(1)
    assert not bad.any(), (a[bad][:3], b[bad][:3], got[bad][:3], want[bad][:3])
    assert np.array_equal(c, (a < b) | (a > 0).astype(np.uint8) << 1 | (a < 0).astype(np.uint8) << 2)
