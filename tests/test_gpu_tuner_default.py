"""The shape the tuner calls the default is the one an untuned solve runs, and
it is among the candidates."""
import numpy as np
import pytest

from conftest import tflows

mesh = tflows.mesh
pytestmark = pytest.mark.gpu


# 230,400 rows: 512 threads in one block per SM (the tuner's own candidates are
# sized by rows per warp); level sweeps: one block of 256 threads per SM
@pytest.mark.parametrize("prec,tiled", [(1, 0), (2, 0)])
def test_default_is_the_untuned_shape(prec, tiled):
    import torch
    tflows.autotune_clear()
    s = mesh.pressure_system(64, 60, 60, perturb=0.2, seed=3, variable_density=True)
    topo = tflows.Topology.from_system(s)
    val, b = torch.from_numpy(s.A[:-1].copy()).cuda(), torch.from_numpy(s.b).cuda()

    def us(**kw):
        best = 1e30
        for _ in range(6):
            x = torch.zeros_like(b)
            r = topo.solve(val, b, x, "cg", prec, 30, 0.0, opts=tflows.options(ic_tiled=tiled, **kw))
            best = min(best, 1e6 * r["seconds"] / 30)
        return best, r

    plain, r0 = us()
    t = topo.autotune(val, b, "cg", prec, opts=tflows.options(ic_tiled=tiled))
    # one shape timed twice: 15 % is several times what such timings differ by
    assert plain / 1.15 <= t["default_us_per_iteration"] <= plain * 1.15, (plain, t)
    tuned, r1 = us(autotune=1)
    assert (r1["block_size"], r1["grid_blocks"]) == (t["block_size"], t["grid_blocks"])
    assert tuned <= 1.15 * plain
    tflows.autotune_clear()
    topo.close()
