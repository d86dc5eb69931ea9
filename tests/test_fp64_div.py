"""The integer FP64 division of the reference-arithmetic kernels against the
host's IEEE division, bit for bit: the same source compiled by the host
compiler, with the reciprocal estimate off by up to three units either way
(the device's instruction is good to one)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HARNESS = r"""
#include "fp64_div.cuh"
extern "C" void divide(const double* a, const double* b, double* q, long n) {
    for (long i = 0; i < n; ++i) q[i] = tflows::div_rn(a[i], b[i]);
}
"""


@pytest.fixture(scope="module", params=[-3, -1, 0, 1, 3])
def divide(request, tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    (d / "h.cpp").write_text(HARNESS)
    so = d / "h.so"
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-x", "c++", f"-DTF_DIV_ESTIMATE_OFF={request.param}",
                    "-I", os.path.join(ROOT, "t-flows-old-compressible_gb300", "csrc"),
                    str(d / "h.cpp"), "-o", str(so)], check=True)
    fn = ctypes.CDLL(str(so)).divide
    p = ctypes.POINTER(ctypes.c_double)

    def run(a, b):
        q = np.empty_like(a)
        fn(a.ctypes.data_as(p), b.ctypes.data_as(p), q.ctypes.data_as(p), ctypes.c_long(a.size))
        return q
    return run


def _check(divide, a, b):
    with np.errstate(all="ignore"):
        want = a / b
    got = divide(a, b)
    same = (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))
    assert same.all(), (a[~same][:3], b[~same][:3], got[~same][:3], want[~same][:3])


def test_any_bit_patterns(divide):
    rng = np.random.default_rng(0)
    a, b = (rng.integers(0, 2**64, 400_000, dtype=np.uint64).view(np.float64) for _ in range(2))
    _check(divide, a, b)


def test_significands_near_powers_and_of_few_bits(divide):
    rng = np.random.default_rng(1)
    one = np.uint64(1) << np.uint64(52)
    near = [rng.integers(0, 8, 4000, dtype=np.uint64), one - np.uint64(1) - rng.integers(0, 8, 4000, dtype=np.uint64),
            rng.integers(0, 2**23, 4000, dtype=np.uint64) << np.uint64(29),
            (rng.integers(0, 2**23, 4000, dtype=np.uint64) << np.uint64(29)) | np.uint64(2**29 - 1),
            rng.integers(0, 2**52, 4000, dtype=np.uint64)]
    for fa in near:
        for fb in near:
            a = (fa | (np.uint64(1023) << np.uint64(52))).view(np.float64)
            b = (rng.permutation(fb) | (np.uint64(1023) << np.uint64(52))).view(np.float64)
            _check(divide, a, b)


def test_special_operands_and_range_ends(divide):
    s = np.array([0.0, -0.0, 1.0, -3.0, np.inf, -np.inf, np.nan, 5e-324, 2.2250738585072014e-308,
                  4.4e-308, 1e-64, 1.7976931348623157e308, 8.98846567431158e307])
    a, b = (x.ravel().copy() for x in np.meshgrid(s, s))
    _check(divide, a, b)
    rng = np.random.default_rng(2)
    m = rng.uniform(1.0, 2.0, 200_000)
    e = rng.integers(-1021, 1023, 200_000)
    for d in (-1024, -1023, -1022, -1021, 1021, 1022, 1023):  # exponents of the quotient
        k = np.clip(e - d, -1022, 1023)
        _check(divide, np.ldexp(m, np.clip(e, -1022, 1023)), np.ldexp(rng.permutation(m), k))
