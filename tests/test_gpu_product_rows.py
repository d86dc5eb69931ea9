"""The products of the solver loop over the forms of rows they distinguish:
column patterns and explicit columns, slices of one and of several widths,
rows of up to and of more than eight entries, with the search direction
formed inside and before the product."""
import numpy as np
import pytest

from conftest import tflows

pytestmark = pytest.mark.gpu


def _system(n, extra, seed, band):
    """A symmetric positive definite matrix: the offsets `band` on every row
    (few column patterns), or `extra` random neighbours per row on average."""
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    if band:
        a = sp.lil_matrix((n, n))
        for k in band:
            a += sp.diags(rng.uniform(0.5, 1.0, n - k), k, shape=(n, n))
    else:
        m = extra * n // 2
        i, j = rng.integers(0, n, m), rng.integers(0, n, m)
        keep = i < j
        a = sp.coo_matrix((rng.uniform(0.5, 1.0, keep.sum()), (i[keep], j[keep])), shape=(n, n))
    a = sp.csr_matrix(a)
    a = -(a + a.T)
    d = -np.asarray(a.sum(1)).ravel() + rng.uniform(1.0, 2.0, n)
    a = sp.csr_matrix(a + sp.diags(d))
    a.sort_indices()
    return a, rng.uniform(-1, 1, n)


@pytest.mark.parametrize("n", [1, 31, 33, 4097])
@pytest.mark.parametrize("extra,band", [(0, (1, 30)), (0, (1, 2, 3)), (0, (1, 2, 3, 5, 7)), (2, ()),
                                        (12, ())])
@pytest.mark.parametrize("precision,prec,rtol", [("FP64", 1, 1e-12), ("FP64_FMA", 0, 1e-12),
                                                 ("MIXED", 1, 1e-10)])
def test_solves_over_row_forms(n, extra, band, precision, prec, rtol):
    import torch
    a, b = _system(n, extra, n + extra, [k for k in band if k < n])
    rows = np.repeat(np.arange(n), np.diff(a.indptr))
    topo = tflows.Topology(n, a.indptr, a.indices, np.flatnonzero(rows == a.indices))
    val = torch.from_numpy(a.data).cuda()
    bb = torch.from_numpy(b).cuda()
    x = torch.zeros_like(bb)
    tol = rtol * float(np.linalg.norm(b))
    res = topo.solve(val, bb, x, "cg", prec, 2000, tol,
                     opts=tflows.options(precision=getattr(tflows, precision)))
    topo.close()
    assert res["status"] == tflows.OK
    # ||r|| <= tol by the recurrence; the true residual differs from it by
    # the rounding of the iterates, 1e-13 ||b|| here (condition below 100)
    assert np.linalg.norm(b - a @ x.cpu().numpy()) <= tol + 1e-13 * np.linalg.norm(b)
