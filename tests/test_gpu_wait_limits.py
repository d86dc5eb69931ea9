"""Waits that run out inside the IC(0) sweeps and between them: with a limit of
a microsecond, wherever a warp happens to give up, the whole launch ends with
TIMEOUT, and the next solve on the same workspace is unharmed."""
import numpy as np
import pytest

from conftest import tflows

mesh = tflows.mesh
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("tiled", [0, 1])
def test_short_limits_end_the_whole_launch(precision, tiled):
    import torch
    s = mesh.pressure_system(64, 60, 56, perturb=0.2, seed=2, variable_density=True)
    topo = tflows.Topology.from_system(s)
    val, b = torch.from_numpy(s.A[:-1].copy()).cuda(), torch.from_numpy(s.b).cuda()
    kw = {"precision": getattr(tflows, precision), "ic_tiled": tiled, "tol_mode": tflows.TOL_RELATIVE}

    def solve(**more):
        x = torch.zeros_like(b)
        r = topo.solve(val, b, x, "cg", 2, 2000, 1e-10, opts=tflows.options(**kw, **more),
                       raise_on_error=False)
        return r["status"], x.cpu().numpy()

    before = solve()
    assert before[0] == tflows.OK
    for limit in (1e-6, 2e-6, 4e-6, 8e-6, 1.6e-5, 3.2e-5):
        assert solve(timeout_s=limit)[0] in (tflows.TIMEOUT, tflows.OK)
    # the last tile waits some 25 us (116 steps of 0.2 us) for the first one's edges
    assert solve(timeout_s=1e-6)[0] == tflows.TIMEOUT
    after = solve()
    assert after[0] == tflows.OK
    assert np.array_equal(before[1].view(np.uint64), after[1].view(np.uint64))
