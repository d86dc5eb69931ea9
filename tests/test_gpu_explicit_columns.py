"""Mixed solves on both sides of the sizes at which the search direction leaves
the product (500,000 rows with explicit columns, 1.5 million with any): each
reaches its FP64 tolerance, in as many iterations as the same system with column
patterns (to a quarter: the rounding of the reductions decides when a direction
is restarted)."""
import functools
import os

import numpy as np
import pytest

from conftest import tflows

mesh = tflows.mesh
pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=1)
def _pressure(dims):
    return mesh.pressure_system(*dims, perturb=0.2, seed=3, variable_density=True)


# 499,200, 505,600, 1,494,425 and 1,507,650 rows
@pytest.mark.parametrize("dims", [(80, 80, 78), (80, 80, 79), (115, 115, 113), (115, 115, 114)])
@pytest.mark.parametrize("prec,kw", [(0, {}), (1, {}), (1, {"refine_restart": 1}), (2, {"ic_sweeps": 1})])
def test_mixed_solves(dims, prec, kw):
    import torch
    s = _pressure(dims)
    val, b = torch.from_numpy(s.A[:-1].copy()).cuda(), torch.from_numpy(s.b).cuda()
    tol = 1e-8 * float(np.linalg.norm(s.b))
    its = {}
    for patterns in ("1", "0"):
        os.environ["TFLOWS_SELL_PATTERNS"] = patterns
        try:
            topo = tflows.Topology.from_system(s)
        finally:
            del os.environ["TFLOWS_SELL_PATTERNS"]
        assert (topo.patterns > 0) == (patterns == "1")
        x = torch.zeros_like(b)
        r = topo.solve(val, b, x, "cg", prec, 5000, tol, opts=tflows.options(precision=tflows.MIXED, **kw))
        topo.close()
        assert r["status"] == tflows.OK
        # the FP64 residual is tested against tol; formed here in another order (eps ||A|| ||x||)
        assert np.linalg.norm(s.b - s.scipy() @ x.cpu().numpy()) <= tol * (1 + 1e-3)
        its[patterns] = r["inner_iterations"]
    assert abs(its["0"] - its["1"]) <= max(2, its["1"] // 4), its
