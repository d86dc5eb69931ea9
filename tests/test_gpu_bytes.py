"""The algorithmic bytes a solve reports, against the count of what its passes
read and write (a box: column patterns, slices of one width)."""
import pytest

from conftest import tflows

mesh = tflows.mesh
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sweeps", [0, 1, 3])
def test_ic_bytes(sweeps):
    import torch
    s = mesh.pressure_system(24, 20, 18, perturb=0.2, seed=4, variable_density=True)
    topo = tflows.Topology.from_system(s)
    assert topo.patterns > 0
    val, b = torch.from_numpy(s.A[:-1].copy()).cuda(), torch.from_numpy(s.b).cuda()
    x = torch.zeros_like(b)
    r = topo.solve(val, b, x, "cg", 2, 20, 0.0, opts=tflows.options(precision=tflows.FP64_FMA, ic_sweeps=sweeps))
    topo.close()
    n, nnz = s.N, s.NONZ - 1
    off = nnz - n
    product = 8 * nnz + n + 16 * n           # values, a pattern per row, x and y
    if sweeps:
        # per sweep and triangle: its entries, a pattern and a length per row, three vectors
        apply = sweeps * (8 * off + 2 * n * (1 + 4 + 3 * 8))
    else:
        apply = 8 * off + 6 * 8 * n
    its = min(r["iterations"], 20)
    # ten vector accesses per iteration, one fewer with the direction inside the product
    assert r["bytes"] == its * (product + 9 * 8 * n + apply) + product + 4 * 8 * n
