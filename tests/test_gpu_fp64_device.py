"""The integer FP64 arithmetic and the norm test as the GPU runs them, against
the host's IEEE operations bit for bit: any bit patterns, near ties, special
operands beside ordinary ones in every warp, tolerances at the ends of their
range."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from test_fp64_int import SPECIAL, _near

pytestmark = pytest.mark.gpu

HARNESS = r"""
#include "device_common.cuh"
#include "fp64_int.cuh"
using namespace tflows;
__global__ void k(const double* a, const double* b, double* q, unsigned char* c, long n) {
    long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    q[4 * i] = mul_rn(a[i], b[i]);
    q[4 * i + 1] = div_rn(a[i], b[i]);
    q[4 * i + 2] = twice(a[i]);
    q[4 * i + 3] = half(a[i]);
    c[i] = less(a[i], b[i]) | above_zero(a[i]) << 1 | below_zero(a[i]) << 2;
}
__global__ void norms(const double* tol, const double* t, unsigned char* out, long per) {
    __shared__ NormTest n;
    if (threadIdx.x == 0) n.set(tol[blockIdx.x]);
    __syncthreads();
    for (long i = threadIdx.x; i < per; i += blockDim.x)
        out[blockIdx.x * per + i] = n.below(t[blockIdx.x * per + i]);
}
extern "C" int eval(const double* a, const double* b, double* q, unsigned char* c, long n) {
    k<<<(n + 255) / 256, 256>>>(a, b, q, c, n);
    return cudaDeviceSynchronize();
}
extern "C" int below(const double* tol, const double* t, unsigned char* out, long n, long per) {
    norms<<<n, 64>>>(tol, t, out, per);
    return cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("fp64")
    (d / "h.cu").write_text(HARNESS)
    so = d / "h.so"
    subprocess.run([os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc"),
                    "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "t-flows-old-compressible_gb300", "csrc"),
                    str(d / "h.cu"), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("kind", ["any", "near", "mixed"])
def test_products_divisions_and_comparisons(harness, kind):
    import torch
    rng = np.random.default_rng(7)
    if kind == "any":
        a, b = (rng.integers(0, 2**64, 1_000_000, dtype=np.uint64).view(np.float64) for _ in range(2))
    else:
        a, b = _near(rng, 30_000), _near(rng, 30_000)
        b[::7] = a[::7]
        if kind == "mixed":  # special operands in every warp
            a[::5] = rng.choice(SPECIAL, a[::5].size)
            b[::3] = rng.choice(SPECIAL, b[::3].size)
    da, db = torch.from_numpy(a.copy()).cuda(), torch.from_numpy(b.copy()).cuda()
    q = torch.empty((a.size, 4), dtype=torch.float64, device="cuda")
    c = torch.empty(a.size, dtype=torch.uint8, device="cuda")
    assert harness.eval(_ptr(da), _ptr(db), _ptr(q), _ptr(c), ctypes.c_long(a.size)) == 0
    with np.errstate(all="ignore"):
        want = np.column_stack([a * b, a / b, 2.0 * a, 0.5 * a])
    got = q.cpu().numpy()
    same = (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))
    bad = ~same.all(1)
    assert not bad.any(), (a[bad][:3], b[bad][:3], got[bad][:3], want[bad][:3])
    assert np.array_equal(c.cpu().numpy(), (a < b) | (a > 0).astype(np.uint8) << 1 | (a < 0).astype(np.uint8) << 2)


def test_norm_test_is_the_comparison_of_the_root(harness):
    import torch
    rng = np.random.default_rng(8)
    tol = np.concatenate([[0.0, -0.0, -1.0, np.nan, np.inf, -np.inf, 5e-324, 1e-310, 1e-300, 1e-160, 9.9e-141, 1e-140,
                           1.1e-140, 1e-64, 1.0, 3.0, 9.9e139, 1e140, 1.1e140, 1e154, 1.4e154, 1e300, 1.7e308],
                          rng.uniform(1, 10, 200) * 10.0 ** rng.integers(-30, 30, 200)])
    with np.errstate(all="ignore"):
        sq = tol * tol
        around = [sq]
        up = down = sq
        for _ in range(4):
            up, down = np.nextafter(up, np.inf), np.nextafter(down, -np.inf)
            around += [up, down]
        other = [np.full_like(tol, v) for v in (0.0, 5e-324, 1e-300, 1.0, 1e300, 1.7976931348623157e308, np.inf, np.nan)]
        t = np.ascontiguousarray(np.abs(np.stack(around + other, 1)))  # sums of squares
        want = np.sqrt(t) < tol[:, None]
    out = torch.empty(t.shape, dtype=torch.uint8, device="cuda")
    dt, dtol = torch.from_numpy(t).cuda(), torch.from_numpy(tol).cuda()
    assert harness.below(_ptr(dtol), _ptr(dt), _ptr(out), ctypes.c_long(tol.size), ctypes.c_long(t.shape[1])) == 0
    assert np.array_equal(out.cpu().numpy().astype(bool), want)
