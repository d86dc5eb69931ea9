"""Solves on rows of more than eight entries: on both sides of the mean length
at which the FP64 products change their form, lengths that are no multiple of
the entries loaded together, and slices of uneven width."""
import numpy as np
import pytest

from conftest import tflows
from test_gpu_product_rows import _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 4097, 70001])
@pytest.mark.parametrize("extra,band", [(0, 5), (0, 6), (0, 20), (30, 0)])
@pytest.mark.parametrize("method,prec,precision,rtol", [("cg", 1, "FP64", 1e-12), ("cg", 0, "FP64_FMA", 1e-12),
                                                        ("cgs", 1, "FP64", 1e-9), ("cg", 1, "MIXED", 1e-10),
                                                        ("cgs", 1, "MIXED", 1e-10)])
def test_solves_on_long_rows(n, extra, band, method, prec, precision, rtol):
    import torch
    a, b = _system(n, extra, n + extra + band, [k for k in range(1, band + 1) if k < n])
    rows = np.repeat(np.arange(n), np.diff(a.indptr))
    topo = tflows.Topology(n, a.indptr, a.indices, np.flatnonzero(rows == a.indices))
    val, bb = torch.from_numpy(a.data).cuda(), torch.from_numpy(b).cuda()
    x = torch.zeros_like(bb)
    tol = rtol * float(np.linalg.norm(b))
    res = topo.solve(val, bb, x, method, prec, 2000, tol,
                     opts=tflows.options(precision=getattr(tflows, precision)))
    topo.close()
    assert res["status"] == tflows.OK
    # ||r|| <= tol by the recurrence; the true residual differs from it by the
    # rounding of the iterates: 1e-13 ||b|| here (condition below 100), a
    # hundred times that with CGS, whose residual may rise before it falls
    slack = 1e-11 if method == "cgs" else 1e-13
    assert np.linalg.norm(b - a @ x.cpu().numpy()) <= tol + slack * np.linalg.norm(b)
