"""Mixed solves on both sides of the size at which explicit columns take the
search direction out of the product: each reaches its FP64 tolerance, in as
many iterations as the same system with column patterns (to a quarter: the
rounding of the reductions decides when a direction is restarted)."""
import os

import numpy as np
import pytest

from conftest import tflows

mesh = tflows.mesh
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(80, 80, 78), (80, 80, 79)])  # 499,200 and 505,600 rows
@pytest.mark.parametrize("prec,kw", [(0, {}), (1, {}), (1, {"refine_restart": 1}), (2, {"ic_sweeps": 1})])
def test_mixed_solves(dims, prec, kw):
    import torch
    s = mesh.pressure_system(*dims, perturb=0.2, seed=3, variable_density=True)
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
